// SIA velocities on the staggered (Ac) mesh: solve_SIA, ice_dynamics_module.f90:240-314,
// with vertical_integrate / vertical_average (zeta_module.f90:33-85) and map_Ac_to_Aa
// (mesh_ArakawaC_module.f90:770-791).
//
// One thread per Ac edge, columns of the (nAc, nZ) arrays read and written level by level
// (column-major, so each level is a coalesced row of the warp); the Aa average is a small gather
// over iAci. Both are written for few FP64 instructions (the unit that bounds them on GB300).
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "ufe_internal.h"

namespace ufe {

constexpr int kMaxZ = 64;

struct SiaWork {
  int nV = 0, nAc = 0, nZ = 0;
  double *in = nullptr;    // H, sx, sy, sp, so (5 nAc) + A_flow (nAc nZ)
  int *mask = nullptr;     // nAc
  double *out = nullptr;   // D3 (nAc nZ), D, Ux, Uy, Up, Uo (5 nAc), U, V, D Aa (3 nV)
  bool solved = false;
};

void sia_free(SiaWork *w) {
  if (!w) return;
  if (w->in) cudaFree(w->in);
  if (w->mask) cudaFree(w->mask);
  if (w->out) cudaFree(w->out);
  delete w;
}

// Per level, from the host: the factor of A_flow in the integrand (m_enh zeta^n, n = 3) and half the
// distance to the next level.
struct SiaLevels {
  double c[kMaxZ], hdz[kMaxZ];
};

inline SiaLevels sia_levels(const ufe_params *p) {
  SiaLevels l;
  const int n = p->nZ;
  std::memset(&l, 0, sizeof l);
  for (int k = 0; k < n; ++k) {
    l.c[k] = p->m_enh_sia * std::pow(p->zeta[k], 3.0);
    if (k + 1 < n) l.hdz[k] = 0.5 * (p->zeta[k + 1] - p->zeta[k]);
  }
  return l;
}

// One thread per Ac edge. At 2 FP64 lanes a clock per SM the arithmetic, not the 2 * 8 * nZ bytes per
// edge, bounds this kernel: six FP64 instructions per level (the level constants come from the
// host, the sums are fused, the cut-off compares bits) where the direct form takes fifteen. 100k
// vertices (306k edges, 15 levels): 142 -> 57 us, of which 11 are the bytes at the copy rate; 1k: 26 -> 7.7.
// The sums' mean error against extended precision is 2.1e-16, of the direct form 2.5e-16.
template <int NZ>
__global__ void __launch_bounds__(64) k_sia_edges(int nAc, int nZ_rt, const int *__restrict__ mask,
                                                  const double *__restrict__ H, const double *__restrict__ sx,
                                                  const double *__restrict__ sy, const double *__restrict__ sp,
                                                  const double *__restrict__ so, const double *__restrict__ A,
                                                  const __grid_constant__ SiaLevels lev, double *__restrict__ D3,
                                                  double *__restrict__ D, double *__restrict__ Ux,
                                                  double *__restrict__ Uy, double *__restrict__ Up,
                                                  double *__restrict__ Uo) {
  const int nZ = NZ > 0 ? NZ : nZ_rt;
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= nAc) return;
  const size_t ld = (size_t)nAc;
  if (mask[a] == 1) {
    double d3[NZ > 0 ? NZ : kMaxZ];
#pragma unroll
    for (int k = 0; k < nZ; ++k) d3[k] = A[a + (size_t)k * ld];
    const double h = H[a];
    const double p = sp[a], o = so[a];
    const double px = sx[a], py = sy[a];
    // (rho g H)^n * (dHs_dp^2 + dHs_do^2)^((n-1)/2), n = 3: the second power is 1
    const double D0 = (cube_carried((kIceDensity * kGrav) * h) * fma(p, p, o * o)) * (2.0 * h);
    // vertical_integrate( m_enh_sia * A_flow * zeta^n ), from the base upwards; the cut-off and the
    // vertical average on the way
    double f_hi = d3[nZ - 1] * lev.c[nZ - 1];
    double acc = 0.0, avg = 0.0;
    double below = D0 * 0.0;   // the base level (the reference's product with the zero integral)
    d3[nZ - 1] = below;
#pragma unroll
    for (int k = nZ - 2; k >= 0; --k) {
      const double f_lo = d3[k] * lev.c[k];
      acc = fma(-(f_hi + f_lo), lev.hdz[k], acc);
      double v = D0 * acc;
      // below -1e5: a negative number's bits order as its magnitude (NaN stays)
      const long long b = __double_as_longlong(v);
      const unsigned long long m = (unsigned long long)b & 0x7fffffffffffffffull;
      if (b < 0 && m > 0x40f86a0000000000ull && m <= 0x7ff0000000000000ull) v = -1e5;
      d3[k] = v;
      avg = fma(v + below, lev.hdz[k], avg);
      f_hi = f_lo;
      below = v;
    }
    if (D3) {
#pragma unroll
      for (int k = 0; k < nZ; ++k) D3[a + (size_t)k * ld] = d3[k];
    }
    D[a] = h * avg;
    Ux[a] = avg * px;
    Uy[a] = avg * py;
    Up[a] = avg * p;
    Uo[a] = avg * o;
  } else {
    if (D3)
      for (int k = 0; k < nZ; ++k) D3[a + (size_t)k * ld] = 0.0;
    D[a] = 0.0; Ux[a] = 0.0; Uy[a] = 0.0; Up[a] = 0.0; Uo[a] = 0.0;
  }
}

// map_Ac_to_Aa: d_Aa(vi) = sum_ci d_Ac(iAci(vi,ci)) / nC(vi), in ci order; one thread per vertex and
// field (blockIdx.y), each quotient correctly rounded from 1 / nC (divide_by): 3 FP64 instructions
// where a division takes about 20. 1k vertices: 46 -> 6 us; 100k: 138 -> 24 us.
__global__ void __launch_bounds__(128) k_ac_to_aa3(int nV, const int *__restrict__ nC, const int *__restrict__ iAci,
                                                  const double *__restrict__ a0, const double *__restrict__ a1,
                                                  const double *__restrict__ a2, double *__restrict__ b0,
                                                  double *__restrict__ b1, double *__restrict__ b2,
                                                  const __grid_constant__ CountReciprocals rc) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nV) return;
  const double *src = blockIdx.y == 0 ? a0 : blockIdx.y == 1 ? a1 : a2;
  double *dst = blockIdx.y == 0 ? b0 : blockIdx.y == 1 ? b1 : b2;
  const int n = nC[v];
  const double dn = rc.n[n], r = rc.r[n];
  double s = 0.0;
  constexpr int kB = 8;   // values in flight
  for (int c0 = 0; c0 < n; c0 += kB) {
    int e[kB];
    double d[kB];
#pragma unroll
    for (int q = 0; q < kB; ++q) e[q] = c0 + q < n ? iAci[v + (size_t)(c0 + q) * nV] : -1;
#pragma unroll
    for (int q = 0; q < kB; ++q) d[q] = e[q] >= 0 ? src[e[q]] : 0.0;
#pragma unroll
    for (int q = 0; q < kB; ++q)
      if (e[q] >= 0) s = s + divide_by(d[q], dn, r);
  }
  dst[v] = s;
}

// The two launches of a solve.
int launch_sia(const DevMesh &m, const ufe_params *p, const int *mask, const double *H, const double *sx, const double *sy,
               const double *sp, const double *so, const double *A, double *D3, double *D, double *Ux, double *Uy,
               double *Up, double *Uo, double *Ua, double *Va, double *Da, cudaStream_t s) {
  const SiaLevels lev = sia_levels(p);
  const unsigned g = (unsigned)((m.nAc + 63) / 64);
  if (p->nZ == 15)
    k_sia_edges<15><<<g, 64, 0, s>>>(m.nAc, p->nZ, mask, H, sx, sy, sp, so, A, lev, D3, D, Ux, Uy, Up, Uo);
  else
    k_sia_edges<0><<<g, 64, 0, s>>>(m.nAc, p->nZ, mask, H, sx, sy, sp, so, A, lev, D3, D, Ux, Uy, Up, Uo);
  int rc = cuda_status(cudaGetLastError(), "k_sia_edges");
  if (!rc && Ua) {
    static const CountReciprocals counts = count_reciprocals();
    k_ac_to_aa3<<<dim3((unsigned)((m.nV + 127) / 128), 3), 128, 0, s>>>(m.nV, m.nC, m.iAci, Ux, Uy, D, Ua, Va, Da, counts);
    rc = cuda_status(cudaGetLastError(), "k_ac_to_aa3");
  }
  return rc;
}

}  // namespace ufe

using namespace ufe;

namespace ufe {
// Up_SIA_Ac of the last ufe_sia_solve on this handle, on the device, or null.
const double *sia_device_Up(ufe_mesh_h h) {
  const SiaWork *w = h->sia;
  if (!w || !w->solved) return nullptr;
  const size_t na = w->nAc;
  return w->out + na * w->nZ + 3 * na;
}
}  // namespace ufe

namespace ufe {
// ufe_sia_solve; with fields_on_device the mask and the five Ac fields of `in` are device
// arrays of this device (the device geometry preparation), and with A_on_device A_flow_Ac is
// too (the device physical properties); otherwise A_flow_Ac is a host array.
int sia_solve_impl(ufe_mesh_h h, const ufe_params *p, const ufe_sia_in *in, ufe_sia_out *out, bool fields_on_device,
                   bool A_on_device) {
  if (!h || !p || !in || !out) { set_error("ufe_sia_solve: null argument"); return UFE_BAD_ARG; }
  if (!in->mask_sheet_Ac || !in->Hi_Ac || !in->dHs_dx_Ac || !in->dHs_dy_Ac || !in->dHs_dp_Ac ||
      !in->dHs_do_Ac || !in->A_flow_Ac || !p->zeta) {
    set_error("ufe_sia_solve: missing input array");
    return UFE_BAD_ARG;
  }
  if (p->nZ < 2 || p->nZ > kMaxZ) { set_error("ufe_sia_solve: nZ must be in [2, 64]"); return UFE_BAD_ARG; }
  const DevMesh &m = h->m;
  const int nV = m.nV, nAc = m.nAc, nZ = p->nZ;
  cudaStream_t s = h->stream;
  int rc = UFE_OK;
  if (h->sia && h->sia->nZ != nZ) { sia_free(h->sia); h->sia = nullptr; }
  if (!h->sia) {
    SiaWork *w = new SiaWork();
    w->nV = nV; w->nAc = nAc; w->nZ = nZ;
    rc = cuda_status(cudaMalloc(&w->in, ((size_t)5 + nZ) * nAc * sizeof(double)), "sia in");
    if (!rc) rc = cuda_status(cudaMalloc(&w->mask, (size_t)nAc * sizeof(int)), "sia mask");
    if (!rc) rc = cuda_status(cudaMalloc(&w->out, (((size_t)5 + nZ) * nAc + 3 * (size_t)nV) * sizeof(double)), "sia out");
    if (rc) { sia_free(w); return rc; }
    h->sia = w;
  }
  SiaWork *w = h->sia;
  const size_t na = nAc;
  double *H = w->in, *sx = H + na, *sy = sx + na, *sp = sy + na, *so = sp + na, *A = so + na;
  const cudaMemcpyKind kin = fields_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  if (!rc) rc = cuda_status(cudaMemcpyAsync(w->mask, in->mask_sheet_Ac, na * sizeof(int), kin, s), "sia input");
  const double *src[5] = {in->Hi_Ac, in->dHs_dx_Ac, in->dHs_dy_Ac, in->dHs_dp_Ac, in->dHs_do_Ac};
  for (int k = 0; k < 5 && !rc; ++k)
    rc = cuda_status(cudaMemcpyAsync(w->in + k * na, src[k], na * sizeof(double), kin, s), "sia input");
  if (!rc)
    rc = cuda_status(cudaMemcpyAsync(A, in->A_flow_Ac, na * nZ * sizeof(double),
                                     A_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s), "A_flow input");
  double *D3 = w->out, *D = D3 + na * nZ, *Ux = D + na, *Uy = Ux + na, *Up = Uy + na, *Uo = Up + na;
  double *Ua = Uo + na, *Va = Ua + nV, *Da = Va + nV;
  if (!rc) rc = launch_sia(m, p, w->mask, H, sx, sy, sp, so, A, D3, D, Ux, Uy, Up, Uo, Ua, Va, Da, s);
  if (!rc) {
    CopyOut back(s, "D2H");   // the fields' device order
    back.add(out->D_SIA_3D_Ac, D3, na * nZ);
    back.add(out->D_SIA_Ac, D, na);
    back.add(out->Ux_SIA_Ac, Ux, na);
    back.add(out->Uy_SIA_Ac, Uy, na);
    back.add(out->Up_SIA_Ac, Up, na);
    back.add(out->Uo_SIA_Ac, Uo, na);
    back.add(out->U_SIA, Ua, nV);
    back.add(out->V_SIA, Va, nV);
    back.add(out->D_SIA, Da, nV);
    rc = back.flush();
  }
  if (!rc) rc = cuda_status(cudaStreamSynchronize(s), "sia solve");
  w->solved = rc == UFE_OK;
  return rc;
}
}  // namespace ufe

extern "C" int ufe_sia_solve(ufe_mesh_h h, const ufe_params *p, const ufe_sia_in *in, ufe_sia_out *out) {
  return sia_solve_impl(h, p, in, out, false);
}

// ---------------------------------------------------------------------------------------
// solve_SIA without allocation: device-resident inputs and outputs, intermediates in a
// fixed scratch array of this translation unit.
//
// Who needs it: a model that keeps its ice state on the device and reserves its device
// memory up front (its own pool sized to the HBM it wants), and a time loop that must not
// stall: cudaMalloc and cudaFree synchronise the whole device, and the per-handle buffers of
// ufe_sia_solve are (re)allocated on the first call and whenever nZ changes. This entry
// point calls neither; its only device memory beyond the caller's arrays is the scratch
// below, which exists from the moment the module is loaded.
// ---------------------------------------------------------------------------------------
namespace ufe {
namespace {

constexpr int kNoAllocMaxAc = UFE_SIA_NOALLOC_MAX_AC;
constexpr int kNoAllocMaxDevices = 64;
// Layout: D, Ux, Uy, Up, Uo on the Ac edges (kNoAllocMaxAc each), 10 MiB.
constexpr size_t kNoAllocScratch = 5 * (size_t)kNoAllocMaxAc;
static __device__ __align__(256) double g_sia_scratch[kNoAllocScratch];

std::mutex g_scratch_mutex;
double *g_scratch_ptr[kNoAllocMaxDevices] = {};

// Address of the scratch on the current device, looked up once per device.
int scratch_address(int device, double **out) {
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (!g_scratch_ptr[device]) {
    double *p = nullptr;
    const int rc = cuda_status(cudaGetSymbolAddress((void **)&p, g_sia_scratch), "cudaGetSymbolAddress(scratch)");
    if (rc) return rc;
    g_scratch_ptr[device] = p;
  }
  *out = g_scratch_ptr[device];
  return UFE_OK;
}

// The kernels dereference every array given, so each must be device memory of this device
// (or managed memory); a host pointer is rejected here instead of faulting there.
bool on_device(const void *ptr, int device) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, ptr) != cudaSuccess) { cudaGetLastError(); return false; }
  if (at.type == cudaMemoryTypeManaged) return true;
  return at.type == cudaMemoryTypeDevice && at.device == device;
}

}  // namespace
}  // namespace ufe

extern "C" int ufe_sia_solve_noalloc(ufe_mesh_h h, const ufe_params *p, const ufe_sia_in *in, ufe_sia_out *out) {
  if (!h || !p || !in || !out) { set_error("ufe_sia_solve_noalloc: null argument"); return UFE_BAD_ARG; }
  const char *who = "ufe_sia_solve_noalloc";
  if (!in->mask_sheet_Ac || !in->Hi_Ac || !in->dHs_dx_Ac || !in->dHs_dy_Ac || !in->dHs_dp_Ac ||
      !in->dHs_do_Ac || !in->A_flow_Ac || !p->zeta) {
    set_error(std::string(who) + ": missing input array");
    return UFE_BAD_ARG;
  }
  if (p->nZ < 2 || p->nZ > kMaxZ) { set_error(std::string(who) + ": nZ must be in [2, 64]"); return UFE_BAD_ARG; }
  const DevMesh &m = h->m;
  const int nAc = m.nAc;
  if (nAc > kNoAllocMaxAc) {
    char buf[192];
    std::snprintf(buf, sizeof buf, "%s: the mesh has %d Ac edges; the fixed scratch holds at most %d", who, nAc,
                  kNoAllocMaxAc);
    set_error(buf);
    return UFE_BAD_ARG;
  }
  if (!out->U_SIA != !out->V_SIA || !out->U_SIA != !out->D_SIA) {
    set_error(std::string(who) + ": U_SIA, V_SIA and D_SIA are given together or not at all");
    return UFE_BAD_ARG;
  }
  int dev = -1;
  int rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  if (dev != h->device || dev < 0 || dev >= kNoAllocMaxDevices) {
    set_error(std::string(who) + ": the mesh's device must be the current device");
    return UFE_BAD_ARG;
  }
  const void *ins[7] = {in->mask_sheet_Ac, in->Hi_Ac, in->dHs_dx_Ac, in->dHs_dy_Ac, in->dHs_dp_Ac, in->dHs_do_Ac,
                        in->A_flow_Ac};
  const void *outs[9] = {out->D_SIA_3D_Ac, out->D_SIA_Ac, out->Ux_SIA_Ac, out->Uy_SIA_Ac, out->Up_SIA_Ac,
                         out->Uo_SIA_Ac, out->U_SIA, out->V_SIA, out->D_SIA};
  for (const void *q : ins)
    if (!on_device(q, dev)) { set_error(std::string(who) + ": an input array is not device memory of the mesh's device"); return UFE_BAD_ARG; }
  for (const void *q : outs)
    if (q && !on_device(q, dev)) { set_error(std::string(who) + ": an output array is not device memory of the mesh's device"); return UFE_BAD_ARG; }
  double *scratch = nullptr;
  rc = scratch_address(dev, &scratch);
  if (rc) return rc;
  // This call's results live only in the caller's arrays. An earlier ufe_sia_solve's
  // velocities on the handle are now out of date, so they are no longer offered to a
  // thickness update that is given no Up_SIA_Ac (it returns UFE_BAD_ARG instead).
  if (h->sia) h->sia->solved = false;
  cudaStream_t s = h->stream;
  // Ac intermediates the caller did not ask for go to the scratch. Every scratch word a
  // kernel reads is written earlier in the same call, so nothing needs clearing.
  double *edge = scratch;
  const size_t na = nAc;
  double *D = out->D_SIA_Ac ? out->D_SIA_Ac : edge;
  double *Ux = out->Ux_SIA_Ac ? out->Ux_SIA_Ac : edge + na;
  double *Uy = out->Uy_SIA_Ac ? out->Uy_SIA_Ac : edge + 2 * na;
  double *Up = out->Up_SIA_Ac ? out->Up_SIA_Ac : edge + 3 * na;
  double *Uo = out->Uo_SIA_Ac ? out->Uo_SIA_Ac : edge + 4 * na;
  rc = launch_sia(m, p, in->mask_sheet_Ac, in->Hi_Ac, in->dHs_dx_Ac, in->dHs_dy_Ac, in->dHs_dp_Ac, in->dHs_do_Ac,
                    in->A_flow_Ac, out->D_SIA_3D_Ac, D, Ux, Uy, Up, Uo, out->U_SIA, out->V_SIA, out->D_SIA, s);
  if (!rc) rc = cuda_status(cudaStreamSynchronize(s), "sia solve (no allocation)");
  return rc;
}
