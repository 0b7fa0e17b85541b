// Internal declarations shared by the translation units of libufemism_gb300.
#pragma once

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/ufemism_gb300.h"

#ifdef __CUDACC__
#include <cuda_runtime.h>
#else
#include <cuda_runtime_api.h>
#endif

namespace ufe {

constexpr int kMaxDeg = 32;    // neighbours per AaAc row the kernels accept (nconmax <= 31)
constexpr int kSlice = 32;     // rows per SELL slice (one warp, one row per lane)
constexpr int kGroups = 6;     // colours 1..5 (rows swept by SOR), then the edge rows
constexpr int kMaxPatchSlices = 1024;  // slices of 32 rows per patch
// Persistent SSA solver: one spatial patch per CTA, kCtasPerSm CTAs per SM, of kSsaBlock threads on the
// phased sweeps (the halo sweeps: kHaloBlock, ufe_ssa.cu). Measured on the 200k-vertex dome with those:
// 1024 x 1 beats 576 x 2, 640 x 2, 384 x 3 and 320 x 4 for the mixed sweep (more CTAs per SM spill at the
// lower register cap).
#ifndef UFE_SSA_BLOCK
#define UFE_SSA_BLOCK 1024
#endif
#ifndef UFE_SSA_CTAS_PER_SM
#define UFE_SSA_CTAS_PER_SM 1
#endif
constexpr int kSsaBlock = UFE_SSA_BLOCK;
constexpr int kCtasPerSm = UFE_SSA_CTAS_PER_SM;
constexpr int kMaxSync = 64;   // patches one patch may synchronise with

// Physical constants, parameters_module.f90:9-21.
constexpr double kIceDensity = 910.0;
constexpr double kSeawaterDensity = 1028.0;
constexpr double kGrav = 9.81;
constexpr double kPi = 3.141592653589793;

void set_error(const std::string &msg);
int cuda_status(cudaError_t e, const char *what);

void neighbour_functions(double px, double py, int n, const double *qx, const double *qy,
                         bool edge, double *Nx, double *Ny, double *Nxx, double *Nxy,
                         double *Nyy);
int aaac_build(const ufe_base_mesh *b, ufe_aaac_mesh *o, std::string *msg);
// ufe_mesh_create with a chosen number of spatial patches (0: the single-solve default).
int mesh_create(const ufe_mesh_desc *d, int n_patch, ufe_mesh_h *out);

#ifdef __CUDACC__
#define UFE_HD __host__ __device__ __forceinline__
#else
#define UFE_HD inline
#endif
constexpr unsigned kNoCol = 0xffffu;   // no neighbour (16-bit columns of the halo program)
constexpr int kXchBufs = 3;     // exchange buffers, taken in turn by sweep

// A halo program slice's block: eight 16-bit columns per 16-byte piece, then the coefficients
// (mixed: two float2 per piece; FP64: one double2), then per slot the packed row word (local row,
// 0xffff: padding; export number << 16, 0xffff: not exported) and the cross-term coefficient,
// then the row data that change between linear solves (halo_refresh). Boundary slices (edge rows,
// corners) have no coefficients.
struct SliceLayout {
  int coef, row, dat, size;   // byte offsets; the columns come first
};
template <bool kM>
UFE_HD SliceLayout slice_layout(int w, bool boundary) {
  SliceLayout s;
  s.coef = (w > 8 ? (w + 7) / 8 : 1) * 512;
  if (kM) {
    s.row = s.coef + (boundary ? 0 : (w > 6 ? (w + 1) / 2 : 3) * 512);   // at least six entries are read
    s.dat = s.row + 256;           // (local row word, 3 sNxy in FP32)
    s.size = s.dat + 512;          // (1/eu, 1/ev, defect) or (c0 x, c0 y, 1 / count, 0)
  } else {
    s.row = s.coef + (boundary ? 0 : w * 512);
    s.dat = s.row + 512;           // (local row word, 0, cross-term coefficient)
    s.size = s.dat + (boundary ? 0 : 1536);   // fast: 1/e, RHS, -; exact: e, RHS, 1/e
  }
  return s;
}

// Device re-layout of the combined AaAc mesh.
//
// Rows are cut into spatially compact patches (Morton order of the row coordinates), one
// per CTA of the persistent solver. Inside a patch they are permuted into groups: the
// non-edge rows of colour 1, ..., colour 5 (the rows the SOR sweep updates, each colour an
// independent set), then the patch's edge rows (updated by the Neumann boundary condition)
// with corners last. Inside a colour the rows are sorted by degree (descending, stable in
// Morton order) so that the sliced-ELL slices of 32 rows are nearly uniform. Every group
// starts on a multiple of 32; the gaps are padding rows (degree 0) that kernels skip.
struct DevMesh {
  int nV = 0, nAc = 0, nA = 0, ncm = 0;
  int nP = 0;                   // padded device rows
  int nSlices = 0;
  int n_patch = 0;              // spatial patches = CTAs of the persistent SSA solver
  int max_patch_slices = 0;
  int max_sync = 0;
  int n_edge_total = 0;         // edge rows including the four corners
  int bnd_total = 0;            // entries of bnd_nbr
  int64_t nE = 0;               // padded SELL entries

  // Device arrays:
  int *orig_of_dev = nullptr;   // [nP] original 0-based AaAc row, -1 = padding
  int *dev_of_orig = nullptr;   // [nA]
  uint8_t *deg = nullptr;       // [nP]
  int64_t *slice_ptr = nullptr; // [nSlices] first SELL entry of the slice
  int *slice_e0 = nullptr;      // [nSlices] the same as int32
  uint8_t *slice_w = nullptr;   // [nSlices] slice width (entries per row)
  uint8_t *slice_g = nullptr;   // [nSlices] group: colour 0..4, 5 = edge rows
  int *patch_slice = nullptr;   // [n_patch][kGroups + 1] first slice of each group of a patch
  int *patch_edge0 = nullptr;   // [n_patch + 1] first edge ordinal of a patch
  int *edge_row = nullptr;      // [n_edge_total] device row of each edge ordinal
  int *sync_ptr = nullptr;      // [n_patch + 1] CSR of the patches each patch synchronises with
  int *sync_list = nullptr;
  int *col = nullptr;           // [nE] neighbour device row, -1 = padding
  double2 *cuv = nullptr;       // [nE] (4Nxx+Nyy, 4Nyy+Nxx)
  double2 *nxy = nullptr;       // [nE] (Nx, Ny)
  float2 *cuv32 = nullptr;      // [nE]
  float2 *nxy32 = nullptr;      // [nE]
  double2 *h_nxy = nullptr;     // [nP] home (Nx, Ny)
  double2 *h_cuv = nullptr;     // [nP] home (4Nxx+Nyy, 4Nyy+Nxx)
  double *sNxy = nullptr;       // [nP] sum of Nxy over home + neighbours
  double *s3Nxy = nullptr;      // [nP] 3 * sNxy (cross-term coefficient of the fast sweeps)
  float2 *h_nxy32 = nullptr;    // [nP] (Nx, Ny) row sums (home + neighbours), for the mixed viscosity
  float *s3Nxy32 = nullptr;     // [nP] 3 * sNxy in FP32
  // Neumann boundary lists by edge ordinal: edge rows' non-edge neighbours; corners' neighbours
  // with an edge neighbour k encoded as -(k+1).
  int *bnd_ptr = nullptr;       // [n_edge_total + 1]
  int *bnd_nbr = nullptr;
  // Geometry for the po rotation and the GL flux.
  double2 *V = nullptr;         // [nV] vertex x,y
  int2 *Aci12 = nullptr;        // [nAc] (vi, vj) 0-based
  int *iAci = nullptr;          // [nV * ncm] column-major Ac ids (0-based), for map_Ac_to_Aa
  int *nC = nullptr;            // [nV]

  // Halo sweep program (ufe_halo.cuh). One SOR sweep runs in seven phases: colours 1..5, then the
  // edge rows, then the corners. A patch updates, besides its own rows, the halo rows whose
  // updates its own rows read within the same sweep (the closure of "reads a row of an earlier
  // phase"), with the same arithmetic, so that a whole sweep needs the neighbouring patches only
  // once, at its start. Its working copy of the velocities (shared memory) holds its own device
  // rows [p0, p1) at local index p - p0, then its halo rows. The program lists, per phase, slices
  // of 32 slots, one block of columns, coefficients and row data per slice (SliceLayout), in the
  // reference's neighbour order.
  bool has_halo = false;
  int max_local = 0;            // largest own slots + halo rows of a patch
  int max_halo = 0;             // largest number of halo rows of a patch
  int max_hslices = 0;          // largest number of program slices of a patch
  int n_hslices = 0;
  size_t max_hprog32 = 0, max_hprog64 = 0;   // bytes of the largest patch's blocks
  int n_export = 0;             // rows that are another patch's halo rows
  int *hp_slice = nullptr;      // [n_patch * 7 + 1] first program slice of phases 0..6 of each patch, then the end
  int *hp_split = nullptr;      // [n_patch] first slice of phase 0's rows that read halo slots (the others come first)
  uint8_t *hslice_w = nullptr;  // [n_hslices] entries per slot
  int *hslice_b32 = nullptr, *hslice_b64 = nullptr;        // [n_hslices] a slice's block, in 16-byte units
  unsigned char *hprog32 = nullptr, *hprog64 = nullptr;    // the blocks of the mixed and of the FP64 sweeps
  int *hrow_g = nullptr;        // [n_hslices * 32] device row, -1 = padding
  int *hload_ptr = nullptr;     // [n_patch + 1] a patch's halo rows in hload_dev, hload_ex
  int *hload_dev = nullptr;     // device row of each halo slot
  int *hload_ex = nullptr;      // its number among the exported rows
  int *hex_ptr = nullptr;       // [n_patch + 1] a patch's exported rows
};

struct SsaWork;   // per-handle device buffers of the SSA solve (ufe_ssa.cu)
struct SiaWork;   // per-handle device buffers of the SIA solve (ufe_sia.cu)
struct AdjWork;   // per-handle device buffers of the SSA adjoint (ufe_ssa.cu)
struct GeomWork;  // per-handle geometry preparation (ufe_geom.cu)

}  // namespace ufe

struct ufe_mesh_s {
  int device = 0;
  cudaStream_t stream = nullptr;
  int num_sms = 0;
  ufe::DevMesh m;
  ufe::SsaWork *ssa = nullptr;
  ufe::SiaWork *sia = nullptr;
  ufe::AdjWork *adj = nullptr;
  ufe::GeomWork *geom = nullptr;
};

namespace ufe {
// Copies from the device to the caller's arrays, queued on a stream; ranges that continue the one
// before on both sides are one copy (each costs about 20 us from the queue, 80 MB only 460 us).
// A null destination is skipped.
class CopyOut {
 public:
  CopyOut(cudaStream_t s, const char *what) : s_(s), what_(what) {}
  template <class T>
  void add(T *dst, const T *src, size_t n) {
    if (!dst || rc_ || n == 0) return;
    const Range r{reinterpret_cast<char *>(dst), reinterpret_cast<const char *>(src), n * sizeof(T)};
    if (!run_.empty() && (r.dst != run_.back().dst + run_.back().bytes || r.src != run_.back().src + run_.back().bytes)) flush();
    run_.push_back(r);
  }
  int flush() {
    if (!run_.empty() && !rc_) {
      size_t total = 0;
      for (const Range &r : run_) total += r.bytes;
      cudaError_t e = cudaMemcpyAsync(run_[0].dst, run_[0].src, total, cudaMemcpyDeviceToHost, s_);
      if (e == cudaErrorInvalidValue && run_.size() > 1) {   // neighbours that were page-locked separately
        cudaGetLastError();
        e = cudaSuccess;
        for (const Range &r : run_)
          if (e == cudaSuccess) e = cudaMemcpyAsync(r.dst, r.src, r.bytes, cudaMemcpyDeviceToHost, s_);
      }
      rc_ = cuda_status(e, what_);
    }
    run_.clear();
    return rc_;
  }

 private:
  struct Range {
    char *dst;
    const char *src;
    size_t bytes;
  };
  cudaStream_t s_;
  const char *what_;
  std::vector<Range> run_;
  int rc_ = 0;
};

void ssa_free(SsaWork *w);
void sia_free(SiaWork *w);
void adj_free(AdjWork *w);
void geom_free(GeomWork *w);
// ufe_sia_solve with the mask and Ac fields of `in` on the device (A_flow_Ac on the host).
int sia_solve_impl(ufe_mesh_h h, const ufe_params *p, const ufe_sia_in *in, ufe_sia_out *out, bool fields_on_device,
                   bool A_on_device = false);
// Velocities of the last solves on a handle, on the device (caller order), or null.
const double *ssa_device_Up(ufe_mesh_h h);
const double *ssa_device_UV(ufe_mesh_h h);
const double *sia_device_Up(ufe_mesh_h h);
// ufe_ssa_upload from device arrays of this device (sheet_count: grounded-ice vertices).
int ssa_upload_impl(ufe_mesh_h h, const ufe_params *p, const ufe_ssa_in *in, const ufe_ssa_inout *io,
                    bool in_on_device, long long sheet_count);

#ifdef __CUDACC__
// a / b rounded to nearest, given r = 1 / b rounded to nearest (Markstein, IBM J. Res. Dev. 34,
// 1990: the quotient corrected once by its exact remainder is the correctly rounded one when
// nothing over- or underflows). Other exponents take the division itself. GB300's FP64 pipe
// (64 cycles a warp instruction on a quarter SM) makes a division cost about 20 of them, this 3.
static __device__ __noinline__ double divide_ieee(double a, double b) { return a / b; }   // kept off the common path

__device__ __forceinline__ double divide_by(double a, double b, double r) {
  const double q = a * r;
  const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7ffu, eq = ((unsigned)__double2hiint(q) >> 20) & 0x7ffu;
  if (ea - 200u < 1600u && eq - 200u < 1600u) return fma(fma(-q, b, a), r, q);
  if (((unsigned long long)__double_as_longlong(a) << 1) == 0ull && eq < 0x7ffu) return q;   // a zero (r finite): exact
  return divide_ieee(a, b);
}

// 1 / b to within a unit in the last place for normal b: two Newton steps (y += y (1 - b y)) from the
// hardware's 20-bit estimate, 4 FP64 instructions.
__device__ __forceinline__ double reciprocal_newton(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  y = fma(y, fma(-b, y, 1.0), y);
  return fma(y, fma(-b, y, 1.0), y);
}

// 1 / b rounded to nearest: a third step from a value within a unit in the last place rounds correctly
// unless all bits of b's significand are set (Markstein, as above); those and extreme exponents take
// the division. 6 FP64 instructions instead of about 20.
__device__ __forceinline__ double reciprocal_rn(double b) {
  const double y = reciprocal_newton(b), z = fma(fma(-b, y, 1.0), y, y);
  const unsigned hi = (unsigned)__double2hiint(b), lo = (unsigned)__double2loint(b);
  if (((hi >> 20) & 0x7ffu) - 200u < 1600u && !(lo == 0xffffffffu && (hi & 0xfffffu) == 0xfffffu)) return z;
  return divide_ieee(1.0, b);
}

// x^3 with the rounding errors of its products carried (below 0.51 ulp); one that overflows is infinite.
__device__ __forceinline__ double cube_carried(double x) {
  const double x2 = x * x, x3 = x2 * x;
  const double c = x3 + fma(fma(x, x, -x2), x, fma(x2, x, -x3));
  return ((unsigned)__double2hiint(x3) & 0x7ff00000u) == 0x7ff00000u ? x3 : c;
}

// 1 / n of the small counts that the kernels divide by, rounded to nearest (a kernel parameter).
struct CountReciprocals {
  double n[kMaxDeg + 1], r[kMaxDeg + 1];   // n as a double, and 1 / n
};
inline CountReciprocals count_reciprocals() {
  CountReciprocals c;
  c.n[0] = c.r[0] = 0.0;
  for (int n = 1; n <= kMaxDeg; ++n) {
    c.n[n] = (double)n;
    c.r[n] = 1.0 / (double)n;
  }
  return c;
}
#endif
}  // namespace ufe
