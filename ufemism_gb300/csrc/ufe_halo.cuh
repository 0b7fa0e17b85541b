// Halo sweeps of the persistent SSA solver (included by ufe_ssa.cu).
//
// A patch updates, besides its own rows, the halo rows whose updates its own rows read within the
// sweep, so a sweep needs the neighbouring patches only at its start. The chain from a patch's
// last update of a row to its neighbour's first use of it, and the latency of the seven phases
// of a sweep, bound the sweep at every size: at 16k vertices the bytes of a sweep would take
// 0.5 us and the arithmetic less. What is done about it:
//
// * Rows that other patches read travel through an exchange buffer as words of 32 data bits and
//   a 32-bit tag, the number of the sweep that wrote them (the tag and the bits it vouches for
//   share a 64-bit access, so no fence, counter or second load stands between the write and the
//   read). A reader polls the very words it needs. Three buffers in turn: a sweep overwrites the
//   words of three sweeps before, and a patch starts a sweep only when every patch has arrived
//   at the sweep before the last (halo_decide), after it read those.
// * A sweep is decided (converged, diverged) one sweep late from a 64-bit arrival word, read by
//   one thread of the fetch warps while the others sweep. The mixed sweeps keep the extra sweep;
//   the FP64 modes, whose sweep counts are the reference's, take it back (hundo holds every own
//   row's value before its last update).
// * A warp loads its next slice's program (columns, coefficients, row data) before the CTA barrier
//   that ends a phase, so a phase starts with its gathers. A slice is stored as one block, read
//   in 16-byte pieces: eight 16-bit columns, two FP32 or one FP64 coefficient pair at a time.
// * Slices are kept in shared memory as far as they fit (halo_stage).
//
// Every update uses the arithmetic, and the neighbour order, of the phased sweeps, so an own row
// gets the same value either way; own rows alone enter the maximum residual.
#pragma once

namespace ufe {

// This CTA's patch of the halo program, in shared memory.
struct HaloSmem {
  int hps[8];                   // first slice of phases 0..6, and the end
  int hsplit;                   // phase 0: slices [hps[0], hsplit) read no halo slot
  int p0, n_own, nh, hl0, ex0;  // own device rows [p0, p0 + n_own), halo slots, first export
  int act[2];                   // the decision taken during a sweep, by parity
  int act_sync;                 // the decision after a barrier
  unsigned long long lag_prev[8];      // each ring slot's arrival word as last read
  unsigned long long wmax[2][32];      // each warp's maximum |res| of a sweep, by parity
  double num[kMaxDeg + 1], rcp_n[kMaxDeg + 1];   // n and 1 / n, for the boundary means
  // per slice: its block's offset in 16-byte units (bit 31: in the shared stage, else in the
  // global program); its width (bit 8: boundary) and, from bit 16, its rows' offset in the block
  // in 16-byte units
  uint2 tab[kMaxPatchSlices];
  // per warp, colour 1's halo-free rows [0], its others [1], colours 2..5 [2..5] and the boundary
  // rows [6]: the first unit's tab entry, the number of units (one every nwarps, [0]: every warp that
  // does not fetch) and the first unit, counted from the patch's first slice
  uint4 sched[7][32];
};
constexpr unsigned kStaged = 1u << 31;

template <bool kM>
__device__ __forceinline__ void load_patch_halo(const SsaArgs &a, int b, HaloSmem &ps) {
  if (threadIdx.x < 8) {
    ps.lag_prev[threadIdx.x] = 0ull;
    ps.hps[threadIdx.x] = a.hp_slice[b * 7 + threadIdx.x];
  }
  if (threadIdx.x == 0) {
    ps.hsplit = a.hp_split[b];
    ps.hl0 = a.hload_ptr[b];
    ps.nh = a.hload_ptr[b + 1] - a.hload_ptr[b];
    ps.ex0 = a.hex_ptr[b];
    const int s0 = a.patch_slice[b * (kGroups + 1)], s1 = a.patch_slice[b * (kGroups + 1) + kGroups];
    ps.p0 = s0 * kSlice;
    ps.n_own = (s1 - s0) * kSlice;
  }
  if (threadIdx.x >= 32 && threadIdx.x <= 32 + kMaxDeg) {
    const int n = (int)threadIdx.x - 32;
    ps.num[n] = (double)n;
    ps.rcp_n[n] = n > 0 ? 1.0 / (double)n : 0.0;
  }
  __syncthreads();
  for (int s = ps.hps[0] + (int)threadIdx.x; s < ps.hps[7]; s += blockDim.x) {
    const int w = a.hslice_w[s];
    const bool boundary = s >= ps.hps[5];
    const int row = kM ? slice_layout<true>(w, boundary).row : slice_layout<false>(w, boundary).row;
    ps.tab[s - ps.hps[0]] = make_uint2((unsigned)a.hslice_b0[s], (unsigned)w | (boundary ? 256u : 0u) | (unsigned)(row / 16) << 16);
  }
  __syncthreads();
}

// The warps' schedules (after halo_stage). Units are dealt round robin over the whole sweep, so that
// where slices are few a phase's warps are others than those of the phase before, which load their
// next unit meanwhile. A phase of few slices costs its warps' chain of instructions, about 600 cycles
// of which the index arithmetic was some 15%: with it tabulated here (and the thread count a constant
// of the compilation) a mixed sweep takes 3.0 us instead of 3.4 at 4k vertices, 11.4 instead of 11.8
// at 200k, an FP64 sweep 51.9 instead of 54.6 at 200k.
__device__ __forceinline__ void halo_schedule(HaloSmem &ps, int nwarps, int nfetch, int per_slice) {
  for (int i = threadIdx.x; i < 7 * nwarps; i += blockDim.x) {
    const int f = i / nwarps, w = i % nwarps;
    const int first = per_slice * ((f == 0 ? ps.hps[0] : f == 1 ? ps.hsplit : ps.hps[f - 1]) - ps.hps[0]);
    const int end = per_slice * ((f == 0 ? ps.hsplit : f == 6 ? ps.hps[7] : ps.hps[f]) - ps.hps[0]);
    const int stride = f == 0 ? nwarps - nfetch : nwarps;
    int u = first + (w - first % nwarps + nwarps) % nwarps;
    if (f == 0) u = w < stride ? first + w : end;
    const int n = u < end ? (end - u + stride - 1) / stride : 0;
    const uint2 t = n ? ps.tab[u / per_slice] : make_uint2(0u, 0u);
    ps.sched[f][w] = make_uint4(t.x, t.y, (unsigned)n, (unsigned)u);
  }
  __syncthreads();
}

// Resident program slices: copies of the patch's slice blocks in the shared memory left after the
// working copy and the halo indices (stage_bytes). All of them when they fit; else the boundary
// slices first (short, and alone in their phases), then whole rounds (a slice per warp) of the colour
// phases, smallest first: the rounds after the first of a colour, whose loads nothing hides (the
// first round's are issued before the barrier), and whole colours of at most one round, as many
// as fit. Thread 0 plans, then the CTA copies the blocks; halo_refresh fills in the row data.
// Warps that fetch the halo slots (the others run colour 1's halo-free rows meanwhile).
__host__ __device__ constexpr int fetch_warps(int nwarps) { return nwarps >= 16 ? 4 : nwarps >= 8 ? 2 : 1; }

template <bool kM>
__device__ void halo_stage(const SsaArgs &a, HaloSmem &ps, unsigned char *stage, int skip_tail) {
  constexpr int kMaxUnits = 64;
  __shared__ int u0[kMaxUnits], u1[kMaxUnits], ub[kMaxUnits];
  const int base = ps.hps[0];
  auto bytes_of = [&](int s) {
    const unsigned y = ps.tab[s - base].y;
    const SliceLayout q = slice_layout<kM>((int)(y & 255u), (y & 256u) != 0);
    return (y & 256u) ? q.size : q.size - skip_tail;
  };
  __syncthreads();
  if (threadIdx.x == 0 && a.stage_bytes > 0) {
    const int nw = (int)(blockDim.x >> 5);
    int nu = 0, used = 0;
    auto unit = [&](int s0, int s1) {
      if (s0 >= s1 || nu >= kMaxUnits) return;
      int b = 0;
      for (int q = s0; q < s1; ++q) b += bytes_of(q);
      u0[nu] = s0; u1[nu] = s1; ub[nu++] = b;
    };
    auto place = [&](int k) {
      for (int q = u0[k]; q < u1[k]; ++q) {
        const int n = bytes_of(q);
        ps.tab[q - base].x = kStaged | (unsigned)(used / 16);
        // (the block's global offset is read again from the program when it is copied)
        used += n;
      }
      ub[k] = -1;
    };
    unit(ps.hps[0], ps.hps[7]);
    if (ub[0] <= a.stage_bytes) {
      place(0);
    } else {
      nu = 0;
      unit(ps.hps[5], ps.hps[7]);
      if (nu && ub[0] <= a.stage_bytes) place(0);
      nu = 0;
      for (int f = -1; f < 5; ++f) {   // -1: colour 1's halo-free rows, 0: its other rows
        const int s0 = f < 0 ? ps.hps[0] : f == 0 ? ps.hsplit : ps.hps[f];
        const int s1 = f < 0 ? ps.hsplit : ps.hps[f + 1];
        const int rs = nw - (f < 0 ? fetch_warps(nw) : 0);
        for (int r = s1 - s0 <= rs ? s0 : s0 + rs; r < s1; r += rs) unit(r, r + rs < s1 ? r + rs : s1);
      }
      for (;;) {
        int best = -1;
        for (int k = 0; k < nu; ++k)
          if (ub[k] >= 0 && (best < 0 || ub[k] < ub[best])) best = k;
        if (best < 0 || used + ub[best] > a.stage_bytes) break;
        place(best);
      }
    }
  }
  __syncthreads();
  const int wid = threadIdx.x >> 5, nwarps = blockDim.x >> 5, lane = threadIdx.x & 31;
  for (int s = base + wid; s < ps.hps[7]; s += nwarps) {
    const unsigned x = ps.tab[s - base].x;
    if (!(x & kStaged)) continue;
    const uint4 *src = reinterpret_cast<const uint4 *>(a.hprog) + a.hslice_b0[s];
    uint4 *dst = reinterpret_cast<uint4 *>(stage) + (x & ~kStaged);
    for (int k = lane; k < bytes_of(s) / 16; k += kSlice) dst[k] = src[k];
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------------------
// Exchange words: 32 data bits and a 32-bit tag in each 64-bit access
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void st_words(unsigned long long *p, unsigned lo, unsigned hi, unsigned tag) {
  const unsigned long long w0 = (unsigned long long)tag << 32 | lo, w1 = (unsigned long long)tag << 32 | hi;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(w0), "l"(w1));
}
__device__ __forceinline__ void ld_words(const unsigned long long *p, unsigned long long &w0, unsigned long long &w1) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(w0), "=l"(w1) : "l"(p));
}
// An exported value: two words (an FP32 pair, or one FP64 component of a row's four words).
__device__ __forceinline__ void export_value(unsigned long long *x, unsigned tag, float2 v) {
  st_words(x, __float_as_uint(v.x), __float_as_uint(v.y), tag);
}
__device__ __forceinline__ void export_value(unsigned long long *x, unsigned tag, double v) {
  st_words(x, (unsigned)__double2loint(v), (unsigned)__double2hiint(v), tag);
}
template <class T> struct XchWords;
template <> struct XchWords<float2> {
  unsigned long long w[2];
  __device__ __forceinline__ void load(const unsigned long long *x, int e) { ld_words(x + 2 * (size_t)e, w[0], w[1]); }
  __device__ __forceinline__ bool ready(unsigned tag) const { return (unsigned)(w[0] >> 32) == tag && (unsigned)(w[1] >> 32) == tag; }
  __device__ __forceinline__ float2 value() const { return make_float2(__uint_as_float((unsigned)w[0]), __uint_as_float((unsigned)w[1])); }
};
template <> struct XchWords<double2> {
  unsigned long long w[4];
  __device__ __forceinline__ void load(const unsigned long long *x, int e) {
    ld_words(x + 4 * (size_t)e, w[0], w[1]);
    ld_words(x + 4 * (size_t)e + 2, w[2], w[3]);
  }
  __device__ __forceinline__ bool ready(unsigned tag) const {
    return (unsigned)(w[0] >> 32) == tag && (unsigned)(w[1] >> 32) == tag && (unsigned)(w[2] >> 32) == tag &&
           (unsigned)(w[3] >> 32) == tag;
  }
  __device__ __forceinline__ double2 value() const {
    return make_double2(__hiloint2double((int)(unsigned)w[1], (int)(unsigned)w[0]),
                        __hiloint2double((int)(unsigned)w[3], (int)(unsigned)w[2]));
  }
};

// A bounded wait's retry: false when the limit has run out (recorded) or another CTA failed.
__device__ __forceinline__ bool wait_retry(const SsaArgs &a, unsigned int *team_bar, unsigned &tries, unsigned long long &t0) {
  if ((++tries & 15u) != 0u) return true;
  if (*(volatile unsigned int *)team_bar & kBarrierError) return false;
  const unsigned long long now = globaltimer_ns();
  if (t0 == 0ull) { t0 = now; return true; }
  if ((long long)(now - t0) > a.timeout_ns) {
    atomicCAS(&a.ctl->err, 0, (int)UFE_TIMEOUT);
    atomicOr(team_bar, kBarrierError);
    return false;
  }
  return true;
}

// The halo slots of the working copy from the exchange, by the last nfetch warps: a thread's
// loads are issued together (kFetchBatch in flight), then repeated until every tag is the sweep's.
template <class T>
__device__ __forceinline__ void halo_poll(const SsaArgs &a, const HaloSmem &ps, const unsigned long long *x,
                                          unsigned tag, unsigned int *team_bar, const int *hidx, T *ld, int nfetch) {
  const int kStride = nfetch * kSlice;
  const int ft = (int)threadIdx.x - ((int)blockDim.x - kStride);
  unsigned tries = 0;
  unsigned long long t0 = 0ull;
  for (int i0 = ft; i0 < ps.nh; i0 += kStride * kFetchBatch) {
    XchWords<T> v[kFetchBatch];
    int e[kFetchBatch];
#pragma unroll
    for (int k = 0; k < kFetchBatch; ++k) {
      const int i = i0 + k * kStride;
      e[k] = i < ps.nh ? hidx[i] : -1;
      if (e[k] >= 0) v[k].load(x, e[k]);
    }
#pragma unroll
    for (int k = 0; k < kFetchBatch; ++k) {
      if (e[k] < 0) continue;
      while (!v[k].ready(tag)) {
        if (!wait_retry(a, team_bar, tries, t0)) return;
        v[k].load(x, e[k]);
      }
      ld[ps.n_own + i0 + k * kStride] = v[k].value();
    }
  }
}

// ---------------------------------------------------------------------------------------
// Colour phases
// ---------------------------------------------------------------------------------------
// What a slice's update needs besides its program, in registers across the sweep.
struct SliceCtx {
  const HaloSmem *ps;
  const unsigned char *stage, *prog;   // the staged and the global slices (mixed: at the lane's 16 bytes)
  unsigned long long *xout;            // this sweep's exchange buffer, at the patch's first export
  unsigned tag;                        // this sweep's tag
  int n_own;
};

__device__ __forceinline__ bool is_dirichlet(const SsaArgs &a, const HaloSmem &ps, int l) {
  return a.skip && a.skip[l < ps.n_own ? ps.p0 + l : a.hload_dev[ps.hl0 + l - ps.n_own]];
}

__device__ __forceinline__ unsigned packed_col(const uint4 &c, int q) {
  const unsigned w = q < 2 ? c.x : q < 4 ? c.y : q < 6 ? c.z : c.w;
  return (q & 1) ? w >> 16 : w & 0xffffu;
}

template <int kMode> struct Prog;

// FP32 correction sweep (as phase_sweep32): a slot a lane. A row's missing entries (beyond its degree)
// name the working copy's zero slot with a coefficient of zero, which leaves the sums unchanged
// (they start at +0 and so are never -0) and needs no test per entry.
template <> struct Prog<kMixed> {
  static constexpr int kPerSlice = 1;   // warps' work units per slice
  uint4 c;
  float4 k[4];
  float4 sd;
  uint2 row;
  uint2 t;

  // b: the block, offset by the lane's 16 bytes
  __device__ __forceinline__ void read(const unsigned char *b) {
    const int w = (int)(t.y & 255u);
    c = *reinterpret_cast<const uint4 *>(b);
    const unsigned char *kp = b + 512;   // the coefficients of slices of up to eight entries
    if (w > 8) kp = b + slice_layout<true>(w, false).coef;
#pragma unroll
    for (int i = 0; i < 3; ++i) k[i] = *reinterpret_cast<const float4 *>(kp + 512 * i);
    if (w > 6) k[3] = *reinterpret_cast<const float4 *>(kp + 3 * 512);
    const unsigned char *r = b + (t.y >> 16) * 16u;
    row = *reinterpret_cast<const uint2 *>(r - (threadIdx.x & 31) * 8);
    sd = *reinterpret_cast<const float4 *>(r + 256);
  }
  __device__ __forceinline__ void load(const SliceCtx &x, uint2 entry, int) {
    t = entry;
    if (t.x & kStaged) read(x.stage + 16u * (t.x & ~kStaged));
    else read(x.prog + 16 * (size_t)t.x);
  }
  __device__ __forceinline__ void update(const SsaArgs &a, const SliceCtx &x, int, float2 *ld, float omega, float &mx) const {
    const unsigned l = row.x & 0xffffu, ex = row.x >> 16;
    if (l == kNoCol) return;   // padding slot
    const float2 di = ld[l];
    if (a.skip && is_dirichlet(a, *x.ps, (int)l)) {
      if (ex != kNoCol) export_value(x.xout + 2 * ex, x.tag, di);
      return;
    }
    float su = 0.0f, sv = 0.0f;
    auto entry = [&](int q) {
      const float2 u = ld[packed_col(c, q)];
      su = fmaf(u.x, (q & 1) ? k[q / 2].z : k[q / 2].x, su);
      sv = fmaf(u.y, (q & 1) ? k[q / 2].w : k[q / 2].y, sv);
    };
#pragma unroll
    for (int q = 0; q < 6; ++q) entry(q);
    const int w = (int)(t.y & 255u);
    if (w > 6) {
      entry(6);
      entry(7);
      if (w > 8) {   // the entries beyond the eighth, from the block
        const unsigned char *b = (t.x & kStaged) ? x.stage + 16u * (t.x & ~kStaged) : x.prog + 16 * (size_t)t.x;
        const SliceLayout y = slice_layout<true>(w, false);
        for (int q = 8; q < w; ++q) {
          const float2 cc = reinterpret_cast<const float2 *>(b + y.coef + (q / 2) * 512)[q % 2];
          const float2 v = ld[reinterpret_cast<const uint16_t *>(b + (q / 8) * 512)[q % 8]];
          su = fmaf(v.x, cc.x, su);
          sv = fmaf(v.y, cc.y, sv);
        }
      }
    }
    const float s3 = __uint_as_float(row.y);
    const float ru = fmaf(fmaf(s3, di.y, su) - sd.z, sd.x, di.x);
    const float rv = fmaf(fmaf(s3, di.x, sv) - sd.w, sd.y, di.y);
    const float2 dn = make_float2(fmaf(-omega, ru, di.x), fmaf(-omega, rv, di.y));
    ld[l] = dn;
    if (ex != kNoCol) export_value(x.xout + 2 * ex, x.tag, dn);
    if ((int)l < x.n_own) mx = max_keep_nan(mx, max_keep_nan(fabsf(ru), fabsf(rv)));
  }
};

// FP64 sweeps (as phase_sweep_fast and phase_sweep_exact). An FP64 instruction occupies a quarter
// SM's unit for 64 cycles (measured), so what counts is how many a warp issues in a row: a lane
// updates one component of one row (16 rows a unit, two units a slice; lanes 0-15 U, 16-31 V),
// which halves a phase's longest chain and spreads a patch's few slices over the four quarters.
template <int kMode> struct Prog {
  static constexpr bool kExact = kMode == kExact64;
  static constexpr int kPerSlice = 2;
  uint4 c;
  double k[8];
  double r, b;        // fast: 1/e, RHS; exact: e, RHS
  double rcp;         // exact: 1/e
  double s3;          // fast: 3 sNxy; exact: sNxy
  unsigned row;
  uint2 t;

  __device__ __forceinline__ void read(const unsigned char *p, int unit) {
    const int w = (int)(t.y & 255u), lane = threadIdx.x & 31;
    const int rl = (unit & 1) * 16 + (lane & 15), rc = 2 * rl + (lane >> 4);
    c = reinterpret_cast<const uint4 *>(p)[rl];
    const double *kp = reinterpret_cast<const double *>(p + (w > 8 ? slice_layout<false>(w, false).coef : 512)) + rc;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < w) k[i] = kp[i * 2 * kSlice];
    const unsigned char *r0 = p + (t.y >> 16) * 16u;
    const uint4 rw = reinterpret_cast<const uint4 *>(r0)[rl];
    row = rw.x;
    s3 = __hiloint2double((int)rw.w, (int)rw.z);
    const double *d = reinterpret_cast<const double *>(r0 + 512) + rc;
    r = d[0];
    b = d[2 * kSlice];
    if (kExact) rcp = d[4 * kSlice];
  }
  __device__ __forceinline__ void load(const SliceCtx &x, uint2 entry, int unit) {
    t = entry;
    if (t.x & kStaged) read(x.stage + 16u * (t.x & ~kStaged), unit);
    else read(x.prog + 16 * (size_t)t.x, unit);
  }
  __device__ __forceinline__ static void add(double u, double cc, double &s) {
    if (kExact) s = s + u * cc;
    else s = fma(u, cc, s);
  }
  __device__ __forceinline__ void update(const SsaArgs &a, const SliceCtx &x, int unit, double2 *ld2, double omega,
                                         unsigned long long &mx) const {
    const unsigned l = row & 0xffffu, ex = row >> 16;
    const int lane = threadIdx.x & 31, comp = lane >> 4, w = (int)(t.y & 255u);
    double *const ld = reinterpret_cast<double *>(ld2) + comp;
    double ui = 0.0, un = 0.0;
    bool put = l != kNoCol;   // padding slots change nothing
    if (put) {
      ui = ld[2 * l];
      const double uo = ld[2 * (int)l + 1 - 2 * comp];   // the row's other component
      un = ui;
      if ((int)l < x.n_own) reinterpret_cast<double *>(a.hundo)[(size_t)64 * x.ps->hps[0] + 32 * unit + 2 * (lane & 15) + comp] = ui;
      if (a.skip && is_dirichlet(a, *x.ps, (int)l)) {
        put = false;
      } else {
        double su = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (q < w) {
            const unsigned j = packed_col(c, q);
            if (j != kNoCol) add(ld[2 * j], k[q], su);
          }
        if (w > 8) {
          const unsigned char *p = (t.x & kStaged) ? x.stage + 16u * (t.x & ~kStaged) : x.prog + 16 * (size_t)t.x;
          const SliceLayout y = slice_layout<false>(w, false);
          const int rl = (unit & 1) * 16 + (lane & 15);
          for (int q = 8; q < w; ++q) {
            const unsigned j = reinterpret_cast<const uint16_t *>(p + (q / 8) * 512 + rl * 16)[q % 8];
            if (j == kNoCol) break;
            add(ld[2 * j], reinterpret_cast<const double *>(p + y.coef)[q * 2 * kSlice + 2 * rl + comp], su);
          }
        }
        double res;
        if (kExact) {
          const double cross = uo * s3;
          const double lhs = (su + 3.0 * cross) + r * ui;
          res = divide_by(lhs - b, r, rcp);
          un = ui - omega * res;
        } else {
          res = fma(fma(s3, uo, su) - b, r, ui);
          un = fma(-omega, res, ui);
        }
        if ((int)l < x.n_own) {
          const unsigned long long bits = abs_bits(res);
          mx = bits > mx ? bits : mx;
        }
      }
    }
    __syncwarp();   // both components of a row are read before either is written
    if (put) ld[2 * l] = un;
    if (l != kNoCol && ex != kNoCol) export_value(x.xout + 4 * ex + 2 * comp, x.tag, un);
  }
};

// ---------------------------------------------------------------------------------------
// Boundary phase f (5: edge rows, 6: corners) of apply_Neumann_boundary_AaAc: the mean of the
// listed neighbours (edge rows: the non-edge ones; corners: all, the edge rows among them already
// updated in phase 5), as phase_boundary. Mixed: c0 + mean of the corrections (phase_boundary).
// FP64: a lane a component, as in the colour phases. The patches with edges and corners run two more
// phases than the others, which wait for them: their first slice's program is loaded before the
// barrier that ends colour 5, by warps dealt as in the colour phases, and the arrival is another
// warp's. The four corner patches' part of a mixed sweep went from 1400 to 920 cycles (4k vertices).
// ---------------------------------------------------------------------------------------
template <int kMode> struct BoundaryProg;

template <> struct BoundaryProg<kMixed> {
  uint4 c;
  float4 c0;      // (c0 x, c0 y, 1 / count, -)
  uint2 t;
  unsigned row;

  __device__ __forceinline__ static const unsigned char *block(const SliceCtx &x, uint2 t) {
    return (t.x & kStaged) ? x.stage + 16u * (t.x & ~kStaged) : x.prog + 16 * (size_t)t.x;
  }
  __device__ __forceinline__ void load(const SliceCtx &x, uint2 entry, int) {
    t = entry;
    const unsigned char *b = block(x, t), *r = b + (t.y >> 16) * 16u;
    c = *reinterpret_cast<const uint4 *>(b);
    row = *reinterpret_cast<const unsigned *>(r - (threadIdx.x & 31) * 8);
    c0 = *reinterpret_cast<const float4 *>(r + 256);
  }
  __device__ __forceinline__ void update(const SsaArgs &, const SliceCtx &x, int, float2 *ld) const {
    const unsigned l = row & 0xffffu, ex = row >> 16;
    if (l == kNoCol) return;
    const int w = (int)(t.y & 255u);
    float sx = 0.0f, sy = 0.0f;
    auto entry = [&](int q) {   // (a row's entries come first)
      const unsigned j = packed_col(c, q);
      if (j != kNoCol) {
        const float2 u = ld[j];
        sx = sx + u.x;
        sy = sy + u.y;
      }
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) entry(q);
    if (w > 4) {
#pragma unroll
      for (int q = 4; q < 8; ++q) entry(q);
      const unsigned char *b = block(x, t);
      for (int q = 8; q < w; ++q) {
        const unsigned j = reinterpret_cast<const uint16_t *>(b + (q / 8) * 512)[q % 8];
        if (j == kNoCol) break;
        const float2 u = ld[j];
        sx = sx + u.x;
        sy = sy + u.y;
      }
    }
    const float2 nv = make_float2(fmaf(sx, c0.z, c0.x), fmaf(sy, c0.z, c0.y));
    ld[l] = nv;
    if (ex != kNoCol) export_value(x.xout + 2 * ex, x.tag, nv);
  }
};

template <int kMode> struct BoundaryProg {
  uint4 c;
  uint2 t;
  unsigned row;

  __device__ __forceinline__ static const unsigned char *block(const SliceCtx &x, uint2 t) {
    return (t.x & kStaged) ? x.stage + 16u * (t.x & ~kStaged) : x.prog + 16 * (size_t)t.x;
  }
  __device__ __forceinline__ void load(const SliceCtx &x, uint2 entry, int unit) {
    t = entry;
    const int rl = (unit & 1) * 16 + (threadIdx.x & 15);
    const unsigned char *b = block(x, t);
    c = reinterpret_cast<const uint4 *>(b)[rl];
    row = reinterpret_cast<const uint4 *>(b + (t.y >> 16) * 16u)[rl].x;
  }
  __device__ __forceinline__ void update(const SsaArgs &a, const SliceCtx &x, int unit, double2 *ld2) const {
    const unsigned l = row & 0xffffu, ex = row >> 16;
    if (l == kNoCol) return;
    const int lane = threadIdx.x & 31, comp = lane >> 4, w = (int)(t.y & 255u), rl = (unit & 1) * 16 + (lane & 15);
    double *const ld = reinterpret_cast<double *>(ld2) + comp;
    double s = 0.0;
    int nvals = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const unsigned j = packed_col(c, q);
      if (j != kNoCol) {
        s = s + ld[2 * j];
        ++nvals;
      }
    }
    if (w > 8) {
      const unsigned char *b = block(x, t);
      for (int q = 8; q < w; ++q) {
        const unsigned j = reinterpret_cast<const uint16_t *>(b + (q / 8) * 512 + rl * 16)[q % 8];
        if (j == kNoCol) break;
        s = s + ld[2 * j];
        ++nvals;
      }
    }
    if (nvals < a.ncm) s = s + 0.0;
    const double nv = divide_by(s, x.ps->num[nvals], x.ps->rcp_n[nvals]);
    if ((int)l < x.n_own) reinterpret_cast<double *>(a.hundo)[(size_t)64 * x.ps->hps[0] + 32 * unit + 2 * (lane & 15) + comp] = ld[2 * l];
    ld[2 * l] = nv;
    if (ex != kNoCol) export_value(x.xout + 4 * ex + 2 * comp, x.tag, nv);
  }
};

// Per-slot copies of the row data a sweep reads that change between linear solves (mixed: the
// FP32 reciprocals of the centre coefficients and the defect; fast FP64: the reciprocals and the
// right-hand side; exact: the centre coefficients, the right-hand side and the reciprocals),
// written into each slice's block by the CTA that reads it, once the grid-wide phase that made
// them is complete.
template <int kMode>
__device__ void halo_refresh(const SsaArgs &a, const HaloSmem &ps, unsigned char *stage) {
  constexpr bool kM = kMode == kMixed;
  for (int k = kSlice * ps.hps[0] + (int)threadIdx.x; k < kSlice * ps.hps[7]; k += blockDim.x) {
    const int g = a.hrow_g[k];
    if (g < 0) continue;
    const int s = k / kSlice, lane = k % kSlice;
    const uint2 t = ps.tab[s - ps.hps[0]];
    const int w = (int)(t.y & 255u);
    const bool boundary = (t.y & 256u) != 0;
    const SliceLayout y = slice_layout<kM>(w, boundary);
    unsigned char *b = (t.x & kStaged) ? stage + 16 * (size_t)(t.x & ~kStaged) : a.hprog + 16 * (size_t)t.x;
    if constexpr (kM) {
      float4 *dat = reinterpret_cast<float4 *>(b + y.dat) + lane;
      if (!boundary) {
        const float2 r = a.rcp32[g], d = a.r0[g];
        *dat = make_float4(r.x, r.y, d.x, d.y);
      } else {
        // c0 = mean of the averaged neighbours' u0 minus the row's u0 (FP64), and 1 / count
        double sx = 0.0, sy = 0.0;
        int n = 0;
        for (int q = 0; q < w; ++q) {
          const unsigned j = reinterpret_cast<const uint16_t *>(b + (q / 8) * 512 + lane * 16)[q % 8];
          if (j == kNoCol) break;
          const double2 u = a.UV[(int)j < ps.n_own ? ps.p0 + (int)j : a.hload_dev[ps.hl0 + (int)j - ps.n_own]];
          sx = sx + u.x;
          sy = sy + u.y;
          ++n;
        }
        const double2 u0 = a.UV[g];
        const double rn = ps.rcp_n[n];
        *dat = make_float4((float)(sx * rn - u0.x), (float)(sy * rn - u0.y), (float)rn, 0.0f);
      }
    } else if (!boundary) {
      // the cross-term coefficient: 3 sNxy, or the parity mode's sNxy
      reinterpret_cast<double *>(b + y.row)[2 * lane + 1] = kMode == kExact64 ? a.sNxy[g] : a.s3Nxy[g];
      double2 *dat = reinterpret_cast<double2 *>(b + y.dat) + lane;
      dat[0] = kMode == kExact64 ? a.euv[g] : a.rcp[g];
      dat[kSlice] = a.rhs[g];
      if (kMode == kExact64) dat[2 * kSlice] = a.rcp[g];
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------------------
// Decisions one sweep late (the words and their ring are those of lag_arrive / lag_decide). No
// data is published under them, so arrivals and reads are relaxed; each CTA's maximum |res| is
// kept per sweep in res_part for the report, read after a barrier.
// ---------------------------------------------------------------------------------------
template <bool kM, class Team>
__device__ __forceinline__ void halo_arrive(const SsaArgs &a, const Team &t, const HaloSmem &ps, unsigned G) {
  // warp 0: the CTA's maximum from the warps' (written before the last barrier)
  const int lane = threadIdx.x & 31;
  unsigned long long x = lane < (int)(blockDim.x >> 5) ? ps.wmax[G & 1][lane] : 0ull;
  if (kM) x = (unsigned long long)__reduce_max_sync(0xffffffffu, (unsigned)x);
  else x = warp_max_u64(x);
  if (lane == 0) {
    unsigned long long inc = 1ull;
    if (kM) {
      const float r = __uint_as_float((unsigned)x);
      if (!(r < a.tol32)) inc += 1ull << 16;
      if (r > 1e6f) inc += 1ull << 32;
      if (r != r) inc += 1ull << 48;
      a.res_part[(G % kLagRing) * t.size() + t.rank()] = (double)r;
    } else {
      const double r = __longlong_as_double((long long)x);
      if (!(r < a.tol)) inc += 1ull << 16;
      if (r > 1e6) inc += 1ull << 32;
      if (r != r) inc += 1ull << 48;
      a.res_part[(G % kLagRing) * t.size() + t.rank()] = r;
    }
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(&a.ctl->lag_word[G % kLagRing]), "l"(inc) : "memory");
  }
}

__device__ __forceinline__ unsigned long long halo_word(const SsaArgs &a, unsigned G) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&a.ctl->lag_word[G % kLagRing]));
  return v;
}

// One thread: the decision on sweep G (1 converged, 2 diverged, 0 neither, -1 a wait failed), its
// word already read once.
template <class Team>
__device__ __forceinline__ int halo_decide(const SsaArgs &a, const Team &t, HaloSmem &ps, unsigned G,
                                           unsigned long long word) {
  const unsigned slot = G % kLagRing;
  const unsigned long long n = (unsigned long long)t.size(), prev = ps.lag_prev[slot];
  unsigned tries = 0;
  unsigned long long t0 = 0ull, d = word - prev;
  while ((d & 0xffffull) < n) {
    if (!wait_retry(a, t.bar(), tries, t0)) return -1;
    d = halo_word(a, G) - prev;
  }
  if ((d & 0xffffull) != n) {   // refilled before it was read (cannot happen: see lag_decide)
    atomicCAS(&a.ctl->err, 0, (int)UFE_TIMEOUT);
    atomicOr(t.bar(), kBarrierError);
    return -1;
  }
  ps.lag_prev[slot] = prev + d;
  const unsigned nc = (unsigned)(d >> 16) & 0xffffu, nd = (unsigned)(d >> 32) & 0xffffu, nn = (unsigned)(d >> 48);
  return nn ? 0 : nc == 0 ? 1 : nd ? 2 : 0;
}

// The whole solve_SSA of one problem on the halo sweeps, run by the CTAs of a team (each CTA owns
// one patch). Returns false when a bounded wait failed; the error is recorded in the problem's
// control block and the team's barrier counter.
template <int kMode, int kThreads, class Team>
__device__ bool solve_member_halo(const SsaArgs &a, Team &t) {
  constexpr bool kM = kMode == kMixed;
  using T = typename std::conditional<kM, float2, double2>::type;
  using Mx = typename std::conditional<kM, float, unsigned long long>::type;
  using Om = typename std::conditional<kM, float, double>::type;
  constexpr int nwarps = kThreads / 32;
  SsaCtl *ctl = a.ctl;
  const bool leader = t.rank() == 0 && threadIdx.x == 0;
  __shared__ HaloSmem ps;
  extern __shared__ __align__(16) unsigned char ufe_local_rows[];
  __syncthreads();   // batched members: every thread is done with the last member's patch
  load_patch_halo<kM>(a, t.rank(), ps);
  T *const ld = reinterpret_cast<T *>(ufe_local_rows);
  int *const hidx = reinterpret_cast<int *>(ufe_local_rows + (size_t)a.halo_index_off);
  unsigned char *const stage = ufe_local_rows + (size_t)a.stage_off;
  for (int i = threadIdx.x; i < ps.nh; i += blockDim.x) hidx[i] = a.hload_ex[ps.hl0 + i];
  halo_stage<kM>(a, ps, stage, kMode == kFast64 ? 512 : 0);
  constexpr int kU = Prog<kMode>::kPerSlice;
  halo_schedule(ps, nwarps, fetch_warps(nwarps), kU);
  const int wid = threadIdx.x >> 5;
  constexpr int nfetch = fetch_warps(nwarps);
  const int decider = (int)blockDim.x - nfetch * kSlice;        // first thread of the fetch warps
  const int n_own = ps.n_own;
  const bool any_boundary = ps.hps[7] > ps.hps[5], any_corners = ps.hps[7] > ps.hps[6];
  const int ex_first = ps.ex0 * (kM ? 2 : 4);
  SliceCtx x{&ps, stage, a.hprog, a.hxch + ex_first, 0u, n_own};
  if (kM) {
    x.stage += 16 * (threadIdx.x & 31);
    x.prog += 16 * (threadIdx.x & 31);
  }
  // the exchange buffers in turn: xout is the next sweep's, xin (for the readers) the last one's
  unsigned long long *xin = a.hxch;
  int turn = 0;
  const T zero{0, 0};
  // The own rows of the working copy: corrections (mixed) start from zero, velocities from UV.
  for (int i = threadIdx.x; i < ps.n_own; i += blockDim.x) {
    if constexpr (kM) ld[i] = zero;
    else ld[i] = a.UV[ps.p0 + i];
  }
  if (threadIdx.x == 0) ld[ps.n_own + ps.nh] = zero;   // the missing entries' slot
  __syncthreads();
  double *N = a.Na, *Nprev = a.Nb;
  int did_reset_before = 0;
  int it = 0;
  unsigned gsweep = 0;   // sweeps of this launch (tags and the decisions' ring)
  bool picard_done = false;
  UFE_TM_DECL
#define UFE_GRID_SYNC() \
  if (!team_barrier(t, &ctl->err, a.timeout_ns)) return false;
  // Mixed: u0 += d, d = 0 on the own rows (each CTA its own; a barrier follows).
  const Om omega = [&]() -> Om { if constexpr (kM) return a.omega32; else return a.omega; }();
  auto fold = [&]() {
    if constexpr (kM) {
      for (int i = threadIdx.x; i < ps.n_own; i += blockDim.x) {
        const float2 d = ld[i];
        if (d.x != 0.0f || d.y != 0.0f) {
          double2 u = a.UV[ps.p0 + i];
          u.x = u.x + (double)d.x;
          u.y = u.y + (double)d.y;
          a.UV[ps.p0 + i] = u;
          ld[i] = zero;
        }
      }
    }
  };
  while (!picard_done && it < a.max_outer) {
    ++it;
    // N_prev <- N, then the new viscosity into N
    { double *q = N; N = Nprev; Nprev = q; }
    phase_viscosity(a, t, N, Nprev, kM && a.fp32_visc, it == 1);
    UFE_GRID_SYNC();
    const double RN = final_rn(a, t);
    if (leader) { ctl->picard_iterations = it; ctl->last_RN = RN; }
    if (RN < a.rn_tol) { picard_done = true; break; }
    phase_coefficients<kMode>(a, t);
    UFE_GRID_SYNC();
    if (kM) {
      phase_defect<true>(a, t);
      UFE_GRID_SYNC();
    }
    int sweeps = 0;
    bool lin_done = false, synced = true;   // synced: a barrier follows the previous sweep, which is decided
    int did_reset = 0;
    int until_refold = a.refold;            // (refold > 0)
    unsigned last_G = 0;                    // the sweep that decided (or ended) the linear solve
    halo_refresh<kMode>(a, ps, stage);
    UFE_TM(kTmOther);
    while (!lin_done && sweeps < a.max_inner) {
      ++sweeps;
      UFE_TM_COUNT(kTmSweeps);
      const unsigned G = gsweep++;
      x.tag = G + 1u;
      Mx mx = 0;
      Prog<kMode> pr;
      // a phase's units of this warp (the first is loaded)
      uint4 sc = make_uint4(0u, 0u, 0u, 0u);
      auto run = [&](int stride) {
        while (sc.z) {
          pr.update(a, x, (int)sc.w, ld, omega, mx);
          if (--sc.z == 0u) break;
          sc.w += (unsigned)stride;
          pr.load(x, ps.tab[sc.w / kU], (int)sc.w);
        }
      };
      auto next = [&](int f) {   // the phase's first unit, loaded before the barrier that the phase waits for
        sc = ps.sched[f][wid];
        if (sc.z) pr.load(x, make_uint2(sc.x, sc.y), (int)sc.w);
      };
      // colour 1's halo-free rows; meanwhile the last warps fetch the halo slots and their first
      // thread the decision on the sweep before
      if (wid < nwarps - nfetch) {
        next(0);
        run(nwarps - nfetch);
      } else if (synced) {
        for (int i = (int)threadIdx.x - decider; i < ps.nh; i += nfetch * kSlice) {
          if constexpr (kM) ld[n_own + i] = zero;
          else ld[n_own + i] = a.UV[a.hload_dev[ps.hl0 + i]];
        }
        if ((int)threadIdx.x == decider) ps.act[G & 1] = 0;
      } else {
        unsigned long long word = 0ull;
        if ((int)threadIdx.x == decider) word = halo_word(a, G - 1u);   // in flight with the halo slots
        halo_poll(a, ps, xin, G, t.bar(), hidx, ld, nfetch);
        if ((int)threadIdx.x == decider) ps.act[G & 1] = halo_decide(a, t, ps, G - 1u, word);
      }
      next(1);
      __syncthreads();
      UFE_TM(kTmWaitColour);
#pragma unroll 1
      for (int f = 1;; ++f) {
        run(nwarps);
        if (f == 5) break;
        next(f + 1);
        __syncthreads();
        UFE_TM_SUB(kTmColour0 + f - 1);
      }
      if constexpr (kM) {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
        if ((threadIdx.x & 31) == 0) ps.wmax[G & 1][wid] = m;
      } else {
        const unsigned long long m = warp_max_u64(mx);
        if ((threadIdx.x & 31) == 0) ps.wmax[G & 1][wid] = m;
      }
      BoundaryProg<kMode> bp;
      if (any_boundary) {
        sc = ps.sched[6][wid];
        if (sc.z) bp.load(x, make_uint2(sc.x, sc.y), (int)sc.w);
      }
      __syncthreads();
      UFE_TM_SUB(kTmColour0 + 4);
      UFE_TM(kTmColour);
      if (wid == nwarps - 1 - nfetch) halo_arrive<kM>(a, t, ps, G);   // (a warp with little else to do)
      UFE_TM(kTmArrive);
      if (any_boundary) {
        // edge rows, then the corners, which average edge rows among others
        auto boundary = [&](unsigned end) {
          while (sc.z && sc.w < end) {
            bp.update(a, x, (int)sc.w, ld);
            sc.w += (unsigned)nwarps;
            if (--sc.z) bp.load(x, ps.tab[sc.w / kU], (int)sc.w);
          }
          __syncthreads();
        };
        boundary((unsigned)(kU * (ps.hps[6] - ps.hps[0])));
        if (any_corners) boundary(~0u);
      }
      // the exchange buffers move on
      xin = x.xout - ex_first;
      turn = turn == kXchBufs - 1 ? 0 : turn + 1;
      x.xout = (turn == 0 ? a.hxch : xin + a.xch_stride) + ex_first;
      UFE_TM(kTmBoundary);
      int act = ps.act[G & 1];
      const bool refold_now = kM && --until_refold == 0;
      synced = false;
      last_G = G;
      if (__builtin_expect(act == 0 && sweeps != a.max_inner && !refold_now, 1)) {
        UFE_TM(kTmOther);
        continue;
      }
      if (act < 0) return false;
      if (refold_now) until_refold = a.refold;
      if (act != 0) {
        last_G = G - 1u;
        if constexpr (!kM) {
          // the sweep after the deciding one is taken back
          --sweeps;
          for (int k = kSlice * ps.hps[0] + (int)threadIdx.x; k < kSlice * ps.hps[7]; k += blockDim.x) {
            const int g = a.hrow_g[k];
            if (g >= ps.p0 && g < ps.p0 + ps.n_own) ld[g - ps.p0] = a.hundo[k];
          }
          __syncthreads();
        }
      } else if (sweeps == a.max_inner || refold_now) {
        UFE_GRID_SYNC();
        if ((int)threadIdx.x == decider) ps.act_sync = halo_decide(a, t, ps, G, halo_word(a, G));
        __syncthreads();
        act = ps.act_sync;
        if (act < 0) return false;
        synced = true;
      }
      if (act == 1) {
        lin_done = true;
      } else if (act == 2) {
        for (int i = threadIdx.x; i < ps.n_own; i += blockDim.x) {
          a.UV[ps.p0 + i] = make_double2(0.0, 0.0);
          ld[i] = zero;
        }
        did_reset = 1;
        lin_done = true;
      } else if (sweeps == a.max_inner) {
        if (leader) ctl->not_converged += 1;
      } else if (refold_now) {
        fold();
        UFE_GRID_SYNC();
        phase_defect<true>(a, t);
        UFE_GRID_SYNC();
        halo_refresh<kMode>(a, ps, stage);
      }
      UFE_TM(kTmOther);
    }
    // the own rows into UV before the grid-wide phases read it
    if (!did_reset) {
      if constexpr (kM) fold();
      else
        for (int i = threadIdx.x; i < ps.n_own; i += blockDim.x) a.UV[ps.p0 + i] = ld[i];
    }
    UFE_GRID_SYNC();
    // the sweep after the deciding one has arrived too: its word is read without acting
    if ((int)threadIdx.x == decider && !synced) {
      const unsigned slot = (gsweep - 1u) % kLagRing;
      ps.lag_prev[slot] = *(volatile unsigned long long *)&ctl->lag_word[slot];
    }
    UFE_TM(kTmGrid);
    if (t.rank() == 0 && threadIdx.x < 32) {
      const volatile double *rp = a.res_part + (size_t)(last_G % kLagRing) * t.size();
      unsigned long long m = 0ull;
      for (int b = threadIdx.x; b < t.size(); b += 32) {
        const unsigned long long v = abs_bits(rp[b]);
        m = v > m ? v : m;
      }
      m = warp_max_u64(m);
      if (leader) {
        if (ctl->linear_solves < 64) ctl->sweeps[ctl->linear_solves] = sweeps;
        ctl->linear_solves += 1;
        ctl->total_sweeps += sweeps;
        ctl->last_max_residual = __longlong_as_double((long long)m);
        if (did_reset) ctl->resets += 1;
      }
    }
    if (did_reset) {
      if (did_reset_before) {
        if (leader) ctl->status = UFE_DIVERGED;
        break;
      }
      did_reset_before = 1;
    }
  }
  // Final N lives in N; make Na hold it for the scatter.
  if (N != a.Na) {
    const int tid = t.rank() * blockDim.x + threadIdx.x;
    const int nt = t.size() * blockDim.x;
    UFE_GRID_SYNC();
    for (int p = tid; p < a.nP; p += nt) a.Na[p] = N[p];
  }
  UFE_GRID_SYNC();
  UFE_TM(kTmOther);
  UFE_TM_FLUSH();
  return true;
#undef UFE_GRID_SYNC
}

}  // namespace ufe
