// The transposed sweeps of the VJP's GMRES iteration as halo sweeps (included by ufe_ssa.cu).
//
// The phased transposed sweep (ssa_adjoint_sor) waits for the neighbouring patches before each of
// its seven phases and reads every entry through L2 twice in a row: 50 us a sweep at 16k vertices,
// where the FP64 instructions take about 6. Here a patch runs the whole sweep on a working copy in
// shared memory (mu and s of its own rows and of the halo rows whose updates it needs, as in
// ufe_halo.cuh) and exchanges rows with its neighbours once a sweep through tagged words. A launch
// does a fixed number of sweeps (GMRES tests nothing in between), each with an exchange buffer of
// its own, so that no patch can overwrite a word before it is read. The arithmetic and the
// neighbour order of a row are those of adj_phase.
#pragma once

namespace ufe {

constexpr int kAdjSweeps = 8;   // sweeps of one launch at most (exchange buffers)

// A slice's block: eight 16-bit columns per 16-byte piece, per entry and row the pairs
// (c.x, k.x), (c.y, k.y), per row the packed word (local row | export number << 16), then the row data.
struct AdjSliceLayout {
  int coef, row, dat, size;
};
UFE_HD AdjSliceLayout adj_slice_layout(int w, bool boundary) {
  AdjSliceLayout s;
  s.coef = (w > 8 ? (w + 7) / 8 : 1) * 512;
  s.row = s.coef + w * 1024;
  s.dat = s.row + 128;                            // g; colour rows also ee, kh, dinv, alpha (512 each), c3 (256)
  s.size = s.dat + (boundary ? 512 : 5 * 512 + 256);
  return s;
}

struct AdjHaloArgs {
  const int *patch_slice;                          // [patches][kGroups + 1], the device row ranges
  const int *hp_slice, *hp_split;                  // phases: corners, edge rows, colours 5..1
  const int *slice_b0, *slice_w;                   // block in 16-byte units; width | 256 for boundary slices
  const int *hrow_g;
  const int *hload_ptr, *hload_dev, *hload_ex, *hex_ptr;
  unsigned char *prog;
  unsigned long long *xch;                         // kAdjSweeps buffers of xch_stride words
  size_t xch_stride;
  const double2 *alpha;
  const double2 *x;                                // the sweeps start from this
  double2 *y;
  const double2 *from;                             // y = from - (sweeps of x); null: y = sweeps of x
  int use_g, n_sweeps;
  unsigned tag0;                                   // tag of the first sweep (never used before on this handle)
  double omega;
  int s_off, index_off, stage_off, stage_bytes;    // shared memory: mu, then s, halo indices, slices
  unsigned int *flag;                              // [0] error bit of the launch, [1] the error
  long long timeout_ns;
};

struct AdjSmem {
  int hps[8];
  int hsplit, p0, n_own, nh, hl0, ex0;
  uint2 tab[kMaxPatchSlices];
};

struct AdjProg {
  uint4 c;
  double2 k[8];
  double ee, kh, dinv, g, c3, ax, ay;
  unsigned row;
  uint2 t;

  __device__ __forceinline__ const unsigned char *block(const AdjHaloArgs &a, const unsigned char *stage) const {
    return (t.x & kStaged) ? stage + 16 * (size_t)(t.x & ~kStaged) : a.prog + 16 * (size_t)t.x;
  }
  __device__ __forceinline__ void load(const AdjHaloArgs &a, const AdjSmem &ps, const unsigned char *stage, int unit) {
    t = ps.tab[(unit >> 1) - ps.hps[0]];
    const int w = (int)(t.y & 255u), lane = threadIdx.x & 31;
    const bool boundary = (t.y & 256u) != 0;
    const int rl = (unit & 1) * 16 + (lane & 15), rc = 2 * rl + (lane >> 4);
    const AdjSliceLayout q = adj_slice_layout(w, boundary);
    const unsigned char *p = block(a, stage);
    c = reinterpret_cast<const uint4 *>(p)[rl];
    const double2 *kp = reinterpret_cast<const double2 *>(p + q.coef) + rc;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < w) k[i] = kp[i * 2 * kSlice];
    row = reinterpret_cast<const unsigned *>(p + q.row)[rl];
    const double *d = reinterpret_cast<const double *>(p + q.dat);
    g = a.use_g ? d[rc] : 0.0;
    if (!boundary) {
      ee = d[64 + rc];
      kh = d[128 + rc];
      dinv = d[192 + rc];
      ax = d[256 + 2 * rl];
      ay = d[256 + 2 * rl + 1];
      c3 = d[320 + rl];
    }
  }
  // One component of 16 rows' updates (lanes 0-15 x, 16-31 y).
  __device__ __forceinline__ void update(const AdjHaloArgs &a, const AdjSmem &ps, const unsigned char *stage, int unit,
                                         double *mu2, double *sv, unsigned long long *xout, unsigned tag) const {
    const unsigned l = row & 0xffffu, ex = row >> 16;
    const int lane = threadIdx.x & 31, comp = lane >> 4, w = (int)(t.y & 255u);
    const bool live = l != kNoCol, boundary = (t.y & 256u) != 0;
    double *const mu = mu2 + comp;
    double mn = 0.0;
    if (live) {
      const double mi = mu[2 * l];
      double r = 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < w) {
          const unsigned j = packed_col(c, q);
          if (j != kNoCol) r = fma(k[q].x, mu[2 * j], fma(k[q].y, sv[j], r));
        }
      if (w > 8) {
        const unsigned char *p = block(a, stage);
        const AdjSliceLayout y = adj_slice_layout(w, boundary);
        const int rl = (unit & 1) * 16 + (lane & 15);
        for (int q = 8; q < w; ++q) {
          const unsigned j = reinterpret_cast<const uint16_t *>(p + (q / 8) * 512 + rl * 16)[q % 8];
          if (j == kNoCol) break;
          const double2 cc = reinterpret_cast<const double2 *>(p + y.coef)[q * 2 * kSlice + 2 * rl + comp];
          r = fma(cc.x, mu[2 * j], fma(cc.y, sv[j], r));
        }
      }
      double d;
      if (!boundary) {
        const double mo = mu2[2 * (int)l + 1 - comp];
        r = fma(ee, mi, fma(c3, mo, fma(kh, sv[l], r))) - g;
        d = -a.omega * r * dinv;
      } else {
        d = -(r + mi - g);
      }
      mn = mi + d;
    }
    const double other = __shfl_xor_sync(0xffffffffu, mn, 16);   // (a barrier of the warp's reads, too)
    if (!live) return;
    mu[2 * l] = mn;
    if (ex != kNoCol) export_value(xout + 6 * ex + 2 * comp, tag, mn);
    if (comp == 0) {
      double s = 0.0;
      if (!boundary) {
        s = fma(ax, mn, ay * other);
        sv[l] = s;
      }
      if (ex != kNoCol) export_value(xout + 6 * ex + 4, tag, s);
    }
  }
};

// A bounded wait's retry (as wait_retry); a limit below a microsecond is looked at on every one.
__device__ __forceinline__ bool adj_retry(const AdjHaloArgs &a, unsigned &tries, unsigned long long &t0) {
  if ((++tries & 15u) != 0u && a.timeout_ns >= 1000) return true;
  if (*(volatile unsigned int *)a.flag) return false;
  const unsigned long long now = globaltimer_ns();
  if (t0 == 0ull) { t0 = now; return true; }
  if ((long long)(now - t0) > a.timeout_ns) {
    atomicExch(a.flag + 1, (unsigned)(int)UFE_TIMEOUT);
    atomicExch(a.flag, 1u);
    return false;
  }
  return true;
}

__global__ void __launch_bounds__(kHaloBlock, 1) ssa_adjoint_halo(const __grid_constant__ AdjHaloArgs a) {
  __shared__ AdjSmem ps;
  __shared__ int bad;   // a wait of this CTA failed
  extern __shared__ __align__(16) unsigned char ufe_local_rows[];
  const int b = blockIdx.x;
  if (threadIdx.x < 8) ps.hps[threadIdx.x] = a.hp_slice[b * 7 + threadIdx.x];
  if (threadIdx.x == 0) {
    bad = 0;
    ps.hsplit = a.hp_split[b];
    ps.hl0 = a.hload_ptr[b];
    ps.nh = a.hload_ptr[b + 1] - ps.hl0;
    ps.ex0 = a.hex_ptr[b];
    const int s0 = a.patch_slice[b * (kGroups + 1)], s1 = a.patch_slice[b * (kGroups + 1) + kGroups];
    ps.p0 = s0 * kSlice;
    ps.n_own = (s1 - s0) * kSlice;
  }
  __syncthreads();
  double *const mu = reinterpret_cast<double *>(ufe_local_rows);
  double *const sv = reinterpret_cast<double *>(ufe_local_rows + a.s_off);
  int *const hidx = reinterpret_cast<int *>(ufe_local_rows + a.index_off);
  unsigned char *const stage = ufe_local_rows + a.stage_off;
  const int base = ps.hps[0], nslices = ps.hps[7] - base;
  for (int s = threadIdx.x; s < nslices; s += blockDim.x)
    ps.tab[s] = make_uint2((unsigned)a.slice_b0[base + s], (unsigned)a.slice_w[base + s]);
  __syncthreads();
  // slices into shared memory, first come first served
  if (threadIdx.x == 0) {
    int used = 0;
    for (int s = 0; s < nslices; ++s) {
      const unsigned y = ps.tab[s].y;
      const int n = adj_slice_layout((int)(y & 255u), (y & 256u) != 0).size;
      if (used + n > a.stage_bytes) break;
      ps.tab[s].x = kStaged | (unsigned)(used / 16);
      used += n;
    }
  }
  const double2 *x = a.x;
  for (int i = threadIdx.x; i < ps.n_own + ps.nh; i += blockDim.x) {
    int g = ps.p0 + i;
    if (i >= ps.n_own) {
      g = a.hload_dev[ps.hl0 + i - ps.n_own];
      hidx[i - ps.n_own] = a.hload_ex[ps.hl0 + i - ps.n_own];
    }
    const double2 v = x ? x[g] : make_double2(0.0, 0.0), al = a.alpha[g];
    reinterpret_cast<double2 *>(mu)[i] = v;
    sv[i] = fma(al.x, v.x, al.y * v.y);
  }
  __syncthreads();
  const int wid = threadIdx.x >> 5, nwarps = blockDim.x >> 5, lane = threadIdx.x & 31;
  for (int s = wid; s < nslices; s += nwarps) {
    const uint2 t = ps.tab[s];
    if (!(t.x & kStaged)) continue;
    const uint4 *src = reinterpret_cast<const uint4 *>(a.prog) + a.slice_b0[base + s];
    uint4 *dst = reinterpret_cast<uint4 *>(stage) + (t.x & ~kStaged);
    const int n = adj_slice_layout((int)(t.y & 255u), (t.y & 256u) != 0).size / 16;
    for (int k = lane; k < n; k += kSlice) dst[k] = src[k];
  }
  __syncthreads();
  const int nfetch = fetch_warps(nwarps);
  auto first_unit = [&](int s_begin) { return 2 * s_begin + ((wid - 2 * (s_begin - base)) & (nwarps - 1)); };
  for (int it = 0; it < a.n_sweeps; ++it) {
    unsigned long long *const xout = a.xch + (size_t)it * a.xch_stride + 6 * (size_t)ps.ex0;
    const unsigned tag = a.tag0 + (unsigned)it;
    AdjProg pr;
    // colour 5's rows that read no halo slot, edge row or corner, while the last warps fetch the halo
    if (wid < nwarps - nfetch) {
      for (int u = 2 * ps.hps[2] + wid; u < 2 * ps.hsplit; u += nwarps - nfetch) {
        pr.load(a, ps, stage, u);
        pr.update(a, ps, stage, u, mu, sv, xout, tag);
      }
    } else if (it > 0) {
      const int stride = nfetch * kSlice, ft = (int)threadIdx.x - ((int)blockDim.x - stride);
      const unsigned long long *xin = a.xch + (size_t)(it - 1) * a.xch_stride;
      unsigned tries = 0;
      unsigned long long t0 = 0ull;
      for (int i = ft; i < ps.nh; i += stride) {
        const unsigned long long *q = xin + 6 * (size_t)hidx[i];
        unsigned long long w[6];
        bool ok = true;
        for (;;) {
          ld_words(q, w[0], w[1]);
          ld_words(q + 2, w[2], w[3]);
          ld_words(q + 4, w[4], w[5]);
          bool ready = true;
#pragma unroll
          for (int k = 0; k < 6; ++k) ready = ready && (unsigned)(w[k] >> 32) == tag - 1u;
          if (ready) break;
          if (!adj_retry(a, tries, t0)) { ok = false; break; }
        }
        if (!ok) { bad = 1; break; }
        auto value = [&](int k) { return __hiloint2double((int)(unsigned)w[2 * k + 1], (int)(unsigned)w[2 * k]); };
        reinterpret_cast<double2 *>(mu)[ps.n_own + i] = make_double2(value(0), value(1));
        sv[ps.n_own + i] = value(2);
      }
    }
    int u = first_unit(base);
    if (u < 2 * ps.hps[1]) pr.load(a, ps, stage, u);
    __syncthreads();
    if (bad) return;   // the others notice the flag in their own waits
#pragma unroll 1
    for (int f = 0; f < 7; ++f) {
      const int s_end = ps.hps[f + 1];
      while (u < 2 * s_end) {
        pr.update(a, ps, stage, u, mu, sv, xout, tag);
        u += nwarps;
        if (u < 2 * s_end) pr.load(a, ps, stage, u);
      }
      if (f < 6) {   // the next phase's first unit, before the barrier
        u = first_unit(f == 1 ? ps.hsplit : s_end);
        if (u < 2 * ps.hps[f + 2]) pr.load(a, ps, stage, u);
      }
      if (s_end != ps.hps[f]) __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < ps.n_own; i += blockDim.x) {
    double2 v = reinterpret_cast<const double2 *>(mu)[i];
    if (a.from) {
      const double2 w = a.from[ps.p0 + i];
      v = make_double2(w.x - v.x, w.y - v.y);
    }
    a.y[ps.p0 + i] = v;
  }
}

// The blocks' columns and row words to their places (one warp per slice).
__global__ void k_adj_place(int n_slices, const int *slice_b0, const int *slice_w, const int *index_at, const uint4 *index,
                            unsigned char *prog) {
  const int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (s >= n_slices) return;
  const AdjSliceLayout q = adj_slice_layout(slice_w[s] & 255, (slice_w[s] & 256) != 0);
  uint4 *p = reinterpret_cast<uint4 *>(prog) + slice_b0[s];
  const uint4 *src = index + index_at[s];
  for (int k = lane; k < q.coef / 16; k += 32) p[k] = src[k];
  if (lane < 8) p[q.row / 16 + lane] = src[q.coef / 16 + lane];
}

// The blocks' numbers from the adjoint's set-up kernels (one thread per program slot).
struct AdjFill {
  int n_slots;
  const int *hrow_g, *slice_b0, *slice_w;
  unsigned char *prog;
  const uint8_t *deg;
  const int *slice_e0;
  const double2 *cT, *kT, *ee, *kh, *dinv, *alpha, *g;
  const double *c3;
};
__global__ void k_adj_fill(const AdjFill a) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= a.n_slots) return;
  const int g = a.hrow_g[k];
  if (g < 0) return;
  const int s = k / kSlice, lane = k % kSlice, w = a.slice_w[s] & 255;
  const bool boundary = (a.slice_w[s] & 256) != 0;
  const AdjSliceLayout q = adj_slice_layout(w, boundary);
  unsigned char *p = a.prog + 16 * (size_t)a.slice_b0[s];
  const int n = a.deg[g];
  for (int e = 0; e < n; ++e) {
    const int64_t i = sell_entry(a.slice_e0, g, e);
    const double2 c = a.cT[i], kk = a.kT[i];
    double2 *o = reinterpret_cast<double2 *>(p + q.coef) + e * 2 * kSlice + 2 * lane;
    o[0] = make_double2(c.x, kk.x);
    o[1] = make_double2(c.y, kk.y);
  }
  double2 *d = reinterpret_cast<double2 *>(p + q.dat) + lane;
  d[0] = a.g[g];
  if (!boundary) {
    d[32] = a.ee[g];
    d[64] = a.kh[g];
    d[96] = a.dinv[g];
    d[128] = a.alpha[g];
    reinterpret_cast<double *>(p + q.dat)[320 + lane] = a.c3[g];
  }
}

// ---------------------------------------------------------------------------------------
// Host: the program, built at a handle's first VJP from its device layout
// ---------------------------------------------------------------------------------------
struct AdjHalo {
  bool tried = false, ok = false;
  int n_slices = 0, max_local = 0, max_halo = 0, n_export = 0;
  unsigned tag = 0xffffff00u - 100u;               // next unused tag (near its end, so that every handle passes it early)
  int *ints = nullptr;                             // every index array
  const int *hp_slice = nullptr, *hp_split = nullptr, *slice_b0 = nullptr, *slice_w = nullptr, *hrow_g = nullptr;
  const int *hload_ptr = nullptr, *hload_dev = nullptr, *hload_ex = nullptr, *hex_ptr = nullptr;
  unsigned char *prog = nullptr;
  unsigned long long *xch = nullptr;
  unsigned int *flag = nullptr;
  void free_all() {
    void *p[] = {ints, prog, xch, flag};
    for (void *q : p)
      if (q) cudaFree(q);
    ints = nullptr; prog = nullptr; xch = nullptr; flag = nullptr;
  }
};

// The host's part of the program (no device): from the rows' phases (0 corners, 1 edge rows, 2..6
// colours 5..1, -1 padding) and neighbour lists. False when it does not apply: a working copy or a
// patch too large for the 16-bit columns and the slice table, or a relation that is not symmetric.
struct AdjHaloHost {
  std::vector<int> hp_slice, hp_split, slice_b0, slice_w, hrow_g, hload_ptr, hload_dev, hload_ex, hex_ptr;
  std::vector<unsigned char> index_bytes;          // blocks' columns and row words only, in block order
  std::vector<int> index_at;                       // each slice's first 16-byte unit in index_bytes
  size_t prog_bytes = 0;
  int max_local = 0, max_halo = 0;
};

inline bool adj_build_host(int nP, int n_patch, const std::vector<int> &patch_slice, const std::vector<int8_t> &ph,
                           const std::vector<int> &deg, const std::vector<int> &e0, const std::vector<int> &col,
                           AdjHaloHost &o) {
  auto entry = [&](int p, int k) { return col[(size_t)e0[p / kSlice] + (size_t)k * kSlice + p % kSlice]; };
  auto range = [&](int b, int &p0, int &p1) {
    p0 = patch_slice[(size_t)b * (kGroups + 1)] * kSlice;
    p1 = patch_slice[(size_t)b * (kGroups + 1) + kGroups] * kSlice;
  };
  struct Patch {
    std::vector<int> upd, halo, w, rows, at;       // updated rows, halo rows; slices' widths, rows and index offsets
    std::vector<unsigned char> index;
    int phase[7], split;
  };
  std::vector<Patch> patch(n_patch);
  std::atomic<bool> ok{true};
  // the patches are independent: they are shared out among a few threads
  auto each_patch = [&](auto &&body) {
    const int n = std::max(1, std::min({8, n_patch, (int)std::thread::hardware_concurrency()}));
    std::atomic<int> next{0};
    auto work = [&]() {
      try {
        std::vector<int> mark(nP, -1), other(nP, -1);
        for (int b; (b = next.fetch_add(1)) < n_patch;) body(b, mark, other);
      } catch (...) {                              // out of memory: no program
        ok = false;
      }
    };
    std::vector<std::thread> threads;
    try {
      for (int t = 1; t < n; ++t) threads.emplace_back(work);
    } catch (...) {                                // no more threads: the ones there are do it
    }
    work();
    for (std::thread &t : threads) t.join();
  };
  each_patch([&](int b, std::vector<int> &in_r, std::vector<int> &stamp) {
    int p0, p1;
    range(b, p0, p1);
    std::vector<int> &R = patch[b].upd, &halo = patch[b].halo;
    for (int p = p0; p < p1; ++p)
      if (ph[p] >= 0) {
        in_r[p] = b;
        R.push_back(p);
        for (int k = 0; k < deg[p]; ++k) {         // the relation has to be symmetric
          const int q = entry(p, k);
          bool back = false;
          for (int i = 0; i < deg[q] && !back; ++i) back = entry(q, i) == p;
          if (!back) ok = false;
        }
      }
    for (size_t i = 0; i < R.size(); ++i)
      for (int k = 0; k < deg[R[i]]; ++k) {
        const int j = entry(R[i], k);
        if (ph[j] < ph[R[i]] && in_r[j] != b) { in_r[j] = b; R.push_back(j); }
      }
    auto see = [&](int p) {
      if ((p >= p0 && p < p1) || stamp[p] == b) return;
      stamp[p] = b;
      halo.push_back(p);
    };
    for (int p : R) {
      see(p);
      for (int k = 0; k < deg[p]; ++k) see(entry(p, k));
    }
    std::sort(halo.begin(), halo.end());
    if (p1 - p0 + (int)halo.size() > 65534) ok = false;
  });
  if (!ok) return false;
  std::vector<int> export_of(nP, -1);
  o.hload_ptr.assign(1, 0);
  for (int b = 0; b < n_patch; ++b) {
    int p0, p1;
    range(b, p0, p1);
    const std::vector<int> &halo = patch[b].halo;
    o.max_local = std::max(o.max_local, p1 - p0 + (int)halo.size());
    o.max_halo = std::max(o.max_halo, (int)halo.size());
    o.hload_dev.insert(o.hload_dev.end(), halo.begin(), halo.end());
    o.hload_ptr.push_back((int)o.hload_dev.size());
  }
  for (int p : o.hload_dev) export_of[p] = 0;
  int n_ex = 0;
  for (int b = 0; b < n_patch; ++b) {
    int p0, p1;
    range(b, p0, p1);
    o.hex_ptr.push_back(n_ex);
    for (int p = p0; p < p1; ++p)
      if (export_of[p] == 0) export_of[p] = n_ex++;
  }
  o.hex_ptr.push_back(n_ex);
  o.hload_ex.reserve(o.hload_dev.size());
  for (int p : o.hload_dev) o.hload_ex.push_back(export_of[p]);
  each_patch([&](int b, std::vector<int> &lidx, std::vector<int> &) {
    Patch &q = patch[b];
    int p0, p1;
    range(b, p0, p1);
    const int n_own = p1 - p0;
    for (size_t i = 0; i < q.halo.size(); ++i) lidx[q.halo[i]] = n_own + (int)i;
    auto local_of = [&](int p) { return p >= p0 && p < p1 ? p - p0 : lidx[p]; };
    // rows[7]: colour 5's own rows whose neighbours are own colour rows (they run before the halo is there)
    std::vector<int> rows[8];
    for (int p : q.upd) {
      int f = ph[p];
      if (f == 2 && p >= p0 && p < p1) {
        bool early = true;
        for (int k = 0; k < deg[p] && early; ++k) {
          const int j = entry(p, k);
          early = j >= p0 && j < p1 && ph[j] >= 2;
        }
        if (early) f = 7;
      }
      rows[f].push_back(p);
    }
    for (int step = 0; step < 8; ++step) {
      const int f = step < 2 ? step : step == 2 ? 7 : step - 1;   // corners, edge rows, early colour 5, colours 5..1
      if (f == 2) q.split = (int)q.w.size();
      else q.phase[f == 7 ? 2 : f] = (int)q.w.size();             // phase 2 starts with its early rows
      std::vector<int> &r = rows[f];
      std::stable_sort(r.begin(), r.end(), [&](int x, int y) { return deg[x] > deg[y]; });
      for (size_t s0 = 0; s0 < r.size(); s0 += kSlice) {
        const int n = (int)std::min<size_t>(kSlice, r.size() - s0);
        const int w = deg[r[s0]];
        const AdjSliceLayout y = adj_slice_layout(w, f < 2);
        q.w.push_back(w | (f < 2 ? 256 : 0));
        const size_t at = q.index.size();
        q.at.push_back((int)(at / 16));
        q.index.resize(at + (size_t)y.coef + 128, 0xff);
        uint16_t *cols = reinterpret_cast<uint16_t *>(q.index.data() + at);
        unsigned *words = reinterpret_cast<unsigned *>(q.index.data() + at + y.coef);
        for (int l = 0; l < kSlice; ++l) {
          const int p = l < n ? r[s0 + l] : -1;
          q.rows.push_back(p);
          if (p < 0) continue;
          const unsigned ex = p >= p0 && p < p1 && export_of[p] >= 0 ? (unsigned)(export_of[p] - o.hex_ptr[b]) : kNoCol;
          words[l] = (ex << 16) | (unsigned)local_of(p);
          for (int k = 0; k < deg[p]; ++k) cols[(k / 8) * 256 + l * 8 + k % 8] = (uint16_t)local_of(entry(p, k));
        }
      }
    }
    if ((int)q.w.size() > kMaxPatchSlices) ok = false;
  });
  if (!ok) return false;
  for (const Patch &q : patch) {
    const int first = (int)o.slice_w.size(), index0 = (int)(o.index_bytes.size() / 16);
    for (int f = 0; f < 7; ++f) o.hp_slice.push_back(first + q.phase[f]);
    o.hp_split.push_back(first + q.split);
    for (size_t s = 0; s < q.w.size(); ++s) {
      o.slice_w.push_back(q.w[s]);
      o.slice_b0.push_back((int)(o.prog_bytes / 16));
      o.index_at.push_back(index0 + q.at[s]);
      o.prog_bytes += (size_t)adj_slice_layout(q.w[s] & 255, (q.w[s] & 256) != 0).size;
    }
    o.hrow_g.insert(o.hrow_g.end(), q.rows.begin(), q.rows.end());
    o.index_bytes.insert(o.index_bytes.end(), q.index.begin(), q.index.end());
  }
  o.hp_slice.push_back((int)o.slice_w.size());
  return o.prog_bytes / 16 < ((size_t)1 << 31);
}

// Builds and uploads a handle's program; ok stays false where it does not apply or the device has no
// room for it (the phased sweeps then run).
inline int adj_halo_create(ufe_mesh_h h, AdjHalo &d) {
  d.tried = true;
  const DevMesh &m = h->m;
  cudaStream_t s = h->stream;
  std::vector<int> orig(m.nP), patch_slice((size_t)m.n_patch * (kGroups + 1)), e0(m.nSlices), col((size_t)m.nE), deg(m.nP);
  std::vector<uint8_t> deg8(m.nP), grp(m.nSlices);
  auto down = [&](void *dst, const void *src, size_t n) { return cuda_status(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, s), "adjoint program"); };
  int rc = down(orig.data(), m.orig_of_dev, orig.size() * 4);
  if (!rc) rc = down(patch_slice.data(), m.patch_slice, patch_slice.size() * 4);
  if (!rc) rc = down(e0.data(), m.slice_e0, e0.size() * 4);
  if (!rc) rc = down(col.data(), m.col, col.size() * 4);
  if (!rc) rc = down(deg8.data(), m.deg, deg8.size());
  if (!rc) rc = down(grp.data(), m.slice_g, grp.size());
  if (!rc) rc = cuda_status(cudaStreamSynchronize(s), "adjoint program");
  if (rc) return rc;
  std::vector<int8_t> ph(m.nP, -1);
  for (int p = 0; p < m.nP; ++p) {
    deg[p] = deg8[p];
    if (orig[p] >= 0) ph[p] = (int8_t)(orig[p] < 4 ? 0 : grp[p / kSlice] == 5 ? 1 : 6 - grp[p / kSlice]);
  }
  AdjHaloHost o;
  if (!adj_build_host(m.nP, m.n_patch, patch_slice, ph, deg, e0, col, o)) return UFE_OK;
  // every index array in one allocation
  std::vector<int> all;
  std::vector<size_t> at;
  for (const std::vector<int> *v : {&o.hp_slice, &o.hp_split, &o.slice_b0, &o.slice_w, &o.hrow_g, &o.hload_ptr, &o.hload_dev,
                                    &o.hload_ex, &o.hex_ptr, &o.index_at}) {
    at.push_back(all.size());
    all.insert(all.end(), v->begin(), v->end());
  }
  d.n_slices = (int)o.slice_w.size();
  d.max_local = o.max_local;
  d.max_halo = o.max_halo;
  d.n_export = o.hex_ptr.back();
  const size_t xbytes = (size_t)kAdjSweeps * 6 * d.n_export * sizeof(unsigned long long);
  unsigned char *index = nullptr;
  cudaError_t e = cudaMalloc(&d.ints, all.size() * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&d.prog, o.prog_bytes);
  if (e == cudaSuccess) e = cudaMalloc(&d.xch, xbytes + 16);
  if (e == cudaSuccess) e = cudaMalloc(&d.flag, 2 * sizeof(unsigned int));
  if (e == cudaSuccess) e = cudaMalloc(&index, o.index_bytes.size());
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    d.free_all();
    return UFE_OK;
  }
  rc = cuda_status(e, "adjoint program");
  if (!rc) rc = cuda_status(cudaMemcpyAsync(d.ints, all.data(), all.size() * sizeof(int), cudaMemcpyHostToDevice, s), "adjoint program");
  if (!rc) rc = cuda_status(cudaMemcpyAsync(index, o.index_bytes.data(), o.index_bytes.size(), cudaMemcpyHostToDevice, s), "adjoint program");
  if (!rc) rc = cuda_status(cudaMemsetAsync(d.xch, 0, xbytes + 16, s), "adjoint exchange");
  if (!rc) {
    const int *q = d.ints;
    d.hp_slice = q + at[0]; d.hp_split = q + at[1]; d.slice_b0 = q + at[2]; d.slice_w = q + at[3]; d.hrow_g = q + at[4];
    d.hload_ptr = q + at[5]; d.hload_dev = q + at[6]; d.hload_ex = q + at[7]; d.hex_ptr = q + at[8];
    k_adj_place<<<(unsigned)((d.n_slices + 7) / 8), 256, 0, s>>>(d.n_slices, d.slice_b0, d.slice_w, q + at[9],
                                                                reinterpret_cast<const uint4 *>(index), d.prog);
    rc = cuda_status(cudaGetLastError(), "k_adj_place");
  }
  if (!rc) rc = cuda_status(cudaStreamSynchronize(s), "adjoint program");
  if (index) cudaFree(index);
  if (rc) { d.free_all(); return rc; }
  d.ok = true;
  return UFE_OK;
}

}  // namespace ufe
