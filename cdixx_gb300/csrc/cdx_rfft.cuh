// Register-handoff Stockham engine and the FP32 iteration kernels built on it.
//
// Same transform and pass formula as fft_pass (cdx_fft.cuh), organised so
// that data enter and leave a CTA in registers:
//   * pass 0 loads its butterflies straight from global memory (no staging),
//   * the middle passes exchange through the skewed shared-memory lines,
//   * the last pass leaves its outputs in registers.
// A thread's last-pass outputs of plan 0 are element j + r*NS of line l for
// its butterflies (l, j); the first pass of plan 1 (the radices reversed)
// reads exactly those elements.  So the column pass runs
//     FFT (plan 0) -> projection in registers -> IFFT (plan 1) -> store,
// and the row pass
//     IFFT (plan 0) -> 1/N and update in registers -> FFT (plan 1) -> store,
// with two shared-memory exchanges per 2048-point transform and no staging of
// the lines in or out.
//
// Butterfly g of a pass (g = threadIdx.x + b*T) belongs to line
// l = (g >> cb) & (L-1) and index j = (g >> (cb + log2 L)) << cb | (g & (2^cb - 1)):
// with cb = 0 consecutive threads take consecutive lines (a column tile of
// width L is then read as one contiguous run); the row pass uses cb = log2 of
// the column tile width on tiled data, so 2^cb x L threads cover one piece of
// a tile, and the largest valid cb on row-major data.
// The map is the same for every pass of a kernel, which is what makes the
// register handoff valid.
#pragma once
#include "cdx_kernels.cuh"

namespace cdx {

template <class G, int PLAN, int P>
struct RPass {
  static constexpr int N = G::N;
  static constexpr int R = plan_radix_x(N, PLAN, P);
  static constexpr int NS = plan_ns_x(N, PLAN, P);
  static constexpr int NR = N / R;
  static constexpr int NB = G::L * NR;
  static constexpr int B = (NB + G::T - 1) / G::T;
  static constexpr int TWO = tw_offset_x(N, PLAN, P);
};

// Default butterfly chunk bits of the row pass on column-tiled data: the tile
// width (2^tl threads per tile row piece), except that 8-wide tiles take chunks
// of 16 where the length allows: with chunks of 8 a half-warp spans two lines
// whose stride is 2 mod 16 float2, so its shared-memory accesses conflict
// (512^2: 2.6 M bank conflicts per row pass), while 16 keep each half-warp on
// one line and still read whole 128-byte lines of W.
__host__ __device__ constexpr int row_cb_pick(int tl, int cb_max) {
  return tl == 3 && cb_max >= 4 ? 4 : (tl < cb_max ? tl : cb_max);
}

// largest chunk bits valid for every pass: NR = N / R is a multiple of 2^cb for
// every radix R of the length (both plans have the same radices), so the map
// below is a bijection onto (line, butterfly) in every pass; e.g. 2048 -> 7,
// 192 (NR 12, 48, 64) -> 2, 384 -> 3, 96 -> 1, 48 -> 0
template <int N>
__host__ __device__ constexpr int rfft_cb_max() {
  int c = 0;
  for (;;) {
    for (int p = 0; plan_radix(N, p) != 0; ++p)
      if ((N / plan_radix(N, p)) % (2 << c) != 0) return c;
    ++c;
  }
}

// (l, j) of butterfly b of this thread in a radix-R pass; false past the end
template <class G, int R>
__device__ __forceinline__ bool bfly_of(int b, int cb, int& l, int& j) {
  constexpr int NB = G::L * (G::N / R);
  const int g = threadIdx.x + b * G::T;
  if ((NB % G::T) != 0 && g >= NB) return false;
  l = (g >> cb) & (G::L - 1);
  j = ((g >> (cb + G::LOG2L)) << cb) | (g & ((1 << cb) - 1));
  return true;
}

// Line stride of the row pass in float2.  A half-warp's 16 lanes take chunks of
// 2^cb consecutive columns (cb the default chunk bits) on min(L, 16 / 2^cb) lines,
// 16 / lines columns in all, so lines 16 / lines mod 16 apart put them on 16
// different bank pairs; from cb = 4 on a half-warp stays on one line and the
// column pass's stride (16 / L mod 16 for its line-fastest map) serves both.
// 32, 64, 96, 128 and 384 get a stride of their own; at 48 and 192 the rule gives the
// column pass's (384^2 x32: 60.8 -> 56.0 us per iteration; 192^2 x96 on the 16 lines that
// 256 threads hold 60.9 -> 46.8).
template <class G>
__host__ __device__ constexpr int row_line_stride() {
  constexpr int cb = row_cb_pick(G::LOG2L, rfft_cb_max<G::N>());
  if (cb >= 4) return G::LD;
  const int lines = G::L < (16 >> cb) ? G::L : 16 >> cb;
  return G::BASE + (((16 / lines - G::BASE) % 16) + 16) % 16;
}

// shared-memory word of element i of line l, lines LD words apart
template <int LD>
__device__ __forceinline__ int sidx(int l, int i) { return l * LD + i + (i >> 4); }
// shared-memory word of element j + r*NR of line l (linear in r when NR % 16 == 0)
template <int LD, int NR>
__device__ __forceinline__ int sidx_in(int l, int j, int r) {
  if constexpr (NR % 16 == 0) return sidx<LD>(l, j) + r * (NR + NR / 16);
  else return sidx<LD>(l, j + r * NR);
}
// shared-memory word of element base + r*NS of line l
template <int LD, int R, int NS>
__device__ __forceinline__ int sidx_out(int l, int base, int r) {
  if constexpr (NS % 16 == 0) return sidx<LD>(l, base) + r * (NS + NS / 16);
  else if constexpr (NS == 1 && R == 16) return sidx<LD>(l, base) + r;   // base = 16 j
  else return sidx<LD>(l, base + r * NS);
}

// twiddles and the radix-R DFT of one butterfly of pass P
template <class G, int PLAN, int P, bool INV>
__device__ __forceinline__ void rpass_compute(float2 (&v)[RPass<G, PLAN, P>::R], int j, const float2* tw) {
  using S = RPass<G, PLAN, P>;
  if constexpr (S::NS > 1) {
    const int k = j % S::NS;
#pragma unroll
    for (int r = 1; r < S::R; ++r) {
      float2 w = __ldg(tw + S::TWO + (r - 1) * S::NS + k);
      if (INV) w.y = -w.y;
      v[r] = cmul(v[r], w);
    }
  }
  dftR<S::R, INV>(v);
}

template <class G, int PLAN, int P, int LD>
__device__ __forceinline__ void rpass_store(float2* buf, float2 (&v)[RPass<G, PLAN, P>::B][RPass<G, PLAN, P>::R],
                                            int cb) {
  using S = RPass<G, PLAN, P>;
#pragma unroll
  for (int b = 0; b < S::B; ++b) {
    int l, j;
    if (!bfly_of<G, S::R>(b, cb, l, j)) continue;
    const int k = j % S::NS;
    const int base = (j - k) * S::R + k;
#pragma unroll
    for (int r = 0; r < S::R; ++r) buf[sidx_out<LD, S::R, S::NS>(l, base, r)] = v[b][r];
  }
}

template <class G, int PLAN, int P, int LD>
__device__ __forceinline__ void rpass_load(const float2* buf, float2 (&v)[RPass<G, PLAN, P>::B][RPass<G, PLAN, P>::R],
                                           int cb) {
  using S = RPass<G, PLAN, P>;
#pragma unroll
  for (int b = 0; b < S::B; ++b) {
    int l, j;
    if (!bfly_of<G, S::R>(b, cb, l, j)) continue;
#pragma unroll
    for (int r = 0; r < S::R; ++r) v[b][r] = buf[sidx_in<LD, S::NR>(l, j, r)];
  }
}

template <class G, int PLAN, int P, bool INV>
__device__ __forceinline__ void rpass_compute_all(float2 (&v)[RPass<G, PLAN, P>::B][RPass<G, PLAN, P>::R], int cb,
                                                  const float2* tw) {
  using S = RPass<G, PLAN, P>;
#pragma unroll
  for (int b = 0; b < S::B; ++b) {
    int l, j;
    if (!bfly_of<G, S::R>(b, cb, l, j)) continue;
    rpass_compute<G, PLAN, P, INV>(v[b], j, tw);
  }
}

// middle passes P .. M-2 through shared memory (each ends with a barrier)
template <class G, int PLAN, int P, bool INV, int LD>
__device__ __forceinline__ void rfft_middle(float2* buf, const float2* tw, int cb) {
  if constexpr (P < plan_len(G::N) - 1) {
    using S = RPass<G, PLAN, P>;
    float2 v[S::B][S::R];
    rpass_load<G, PLAN, P, LD>(buf, v, cb);
    __syncthreads();
    rpass_compute_all<G, PLAN, P, INV>(v, cb, tw);
    rpass_store<G, PLAN, P, LD>(buf, v, cb);
    __syncthreads();
    rfft_middle<G, PLAN, P + 1, INV, LD>(buf, tw, cb);
  }
}

template <class G, int PLAN>
using RFirst = RPass<G, PLAN, 0>;
template <class G, int PLAN>
using RLast = RPass<G, PLAN, plan_len(G::N) - 1>;

struct NoHook {
  __device__ __forceinline__ void operator()() const {}
};

// The whole transform of the CTA's L lines: `in` holds pass 0's inputs
// (element j + r*N/R0 of line l for butterfly (l, j)), `out` receives the
// last pass's outputs (element j + r*NS_last).  The shared lines must be free
// on entry (callers synchronise); on return other threads may still be
// reading them, so callers synchronise before the next write.  LD: the line
// stride of `buf` in float2.  `hook` runs
// after every thread's last read of the shared lines has been issued and before
// the last pass's arithmetic (a caller that synchronises there may refill the
// lines while the last pass computes).
template <class G, int PLAN, bool INV, int LD = G::LD, class H = NoHook>
__device__ __forceinline__ void rfft(float2 (&in)[RFirst<G, PLAN>::B][RFirst<G, PLAN>::R],
                                     float2 (&out)[RLast<G, PLAN>::B][RLast<G, PLAN>::R], float2* buf,
                                     const float2* tw, int cb, H&& hook = H{}) {
  constexpr int M = plan_len(G::N);
  rpass_compute_all<G, PLAN, 0, INV>(in, cb, tw);
  if constexpr (M == 1) {
#pragma unroll
    for (int b = 0; b < RFirst<G, PLAN>::B; ++b)
#pragma unroll
      for (int r = 0; r < RFirst<G, PLAN>::R; ++r) out[b][r] = in[b][r];
    hook();
  } else {
    rpass_store<G, PLAN, 0, LD>(buf, in, cb);
    __syncthreads();
    rfft_middle<G, PLAN, 1, INV, LD>(buf, tw, cb);
    rpass_load<G, PLAN, M - 1, LD>(buf, out, cb);
    hook();
    rpass_compute_all<G, PLAN, M - 1, INV>(out, cb, tw);
  }
}

// FP32 launch geometry per length: threads of a CTA (its lines hold about 16 values
// per thread) and the threads per SM its register budget leaves room for.  Small
// CTAs spread a small pattern over more SMs and leave shorter tails; the registers
// (64 a thread at 1024 threads per SM, 80 at 768) trade occupancy for spills.
// Measured, us per iteration, against 256 threads (the geometry of the tensor-core
// modes) at its best budget, L2 warm:
//   64^2 (64 threads)   x1 12.9 -> 10.9, x300 16.7 -> 16.3
//   128^2 (64)          x1 12.2 -> 8.7, x30 13.0 -> 10.5, x100 25.2 -> 17.3, x200 37.3 -> 29.5
//   192^2 (64)          x1 12.6 -> 9.2, x8 13.2 -> 10.3, x96 46.8 -> 42.5
//   256^2 (128)         x1 11.1 -> 9.1, x16 15.1 -> 13.8, x64 39.4 -> 35.5
//   512^2 (128)         x1 11.9 -> 10.5, x16 44.5 -> 43.1, x48 144.3 -> 138.8
//   768^2 (192)         x1 16.4 -> 14.7, x2 23.5 -> 21.7, x8 59.8 -> 54.8
// (1536 on 192: square x1 43.2 -> 42.3, but 768 x 1536 25.0 -> 31.1, so it stays at 256.)
// 192 threads at 768 keep every thread busy in the radix-16 passes.  384
// stays at 256 (96 threads: x1 12.7 -> 12.3 but x8 22.2 -> 23.1, x47 82.6 -> 85.2), as
// do 96 (96 threads: x1 13.3 -> 14.4) and 1024 (128 threads: x4 48.4 -> 50.1) but for
// small work: up to 2^21 pixels a 1024 pass runs on 128 threads with 128 registers
// (1024^2 x1 24.2 -> 17.7, x2 29.4 -> 28.3; use_thin).
constexpr int fp_t(int n) {
  return n == 64 || n == 128 || n == 192 ? 64 : n == 256 || n == 512 ? 128 : n == 768 ? 192 : geom_t(n);
}
constexpr int lines_of(int n, int t) { return pow2_floor(16 * t / n < 2 ? 2 : 16 * t / n); }
template <int N>
struct FGeom : GeomT<N, fp_t(N), lines_of(N, fp_t(N))> {};
constexpr int thin_t(int n) { return n == 1024 ? 128 : fp_t(n); }
template <int N>
struct ThinGeom : GeomT<N, thin_t(N), lines_of(N, thin_t(N))> {};
// threads per SM of the register budget (512 threads and more: two CTAs of 512, else one)
constexpr int res_col(int n, int t) {
  return t >= 512 ? (t == 512 ? 1024 : t) : n == 1024 && t == 128 ? 512 : n == 128 || n == 192 || t == 192 ? 768 : 1024;
}
constexpr int res_row(int n, int t) { return t >= 512 ? t : n >= 1024 && t == 256 ? 768 : res_col(n, t); }

// The row pass stages its rho rows in the line buffer (loading rho straight from
// global memory instead was 4-30 % slower, its latency exposed).
// RHO_IN_BUF: the iterating row pass stages its rho rows in the FFT line buffer
// itself, copied in after the inverse transform's last shared-memory read (the
// copy overlaps the last pass's arithmetic), so the CTA needs one line buffer
// instead of two and four CTAs fit per SM instead of three.
#ifndef CDX_RHO_IN_BUF
#define CDX_RHO_IN_BUF 1
#endif
template <class G>
struct RGeom {
  static constexpr int N = G::N;
  static constexpr bool RHO_IN_BUF = CDX_RHO_IN_BUF && G::T <= 256 && plan_len(N) > 1;
  static constexpr int ROW_LD = row_line_stride<G>();
  static constexpr int SMEM_ROW_LINES = G::L * ROW_LD * (int)sizeof(float2);
  static constexpr int SMEM_ROW_ITER = SMEM_ROW_LINES * (RHO_IN_BUF ? 1 : 2) + G::L * ((N + 31) >> 5) * 4;
  static constexpr int MINB_COL = res_col(N, G::T) / G::T, MINB_ROW = res_row(N, G::T) / G::T;
  static constexpr int MINB_ROW_FFT = G::T == 512 ? 2 : MINB_ROW;
};
// Geometry of a column transform alone whose output is row-major: the default
// tiles of 2 or 4 columns read and write 16- or 32-byte pieces of each row, so the
// lengths from 1024 up take WIDE_L columns in a CTA of WIDE_L N / 16 threads where
// there are enough of them for every SM (whole transform: 4096^2 197 -> 140 us,
// 3072^2 123 -> 95, 2048^2 46.0 -> 37.0, 1024^2 x8 61.7 -> 57.4; 4 columns at 2048^2
// 39.5; 8 at 768^2 x8 35.4 -> 38.3, so 768 keeps its own).  Two CTAs of 512 threads
// per SM in the row transforms of 3072 and 4096 are part of it.
constexpr int wide_l(int n) { return n >= 3072 ? 4 : (n >= 1024 ? 8 : lines_of(n, fp_t(n))); }
template <int N>
struct WideGeom : GeomT<N, wide_l(N) == FGeom<N>::L ? fp_t(N) : wide_l(N) * N / 16, wide_l(N)> {};

// ------------------------------------------------------------- real-space updates
template <int ALGO>
__device__ __forceinline__ float2 update_t(bool inside, float2 x, float2 p, float beta) {
  return apply_update(ALGO, inside, x, p, beta);
}

// ---------------------------------------------------------------- column pass
// Lines are columns (length N = rows).  Column-tiled arrays have tile width L.
// PROJ (COL_ITER): the modulus projection, PROJ_MODABS or PROJ_CCD.
// TL: log2 of the tile width of column-tiled data (COL_FFT on a wide geometry:
// narrower than the CTA's L columns).
template <class G, int MODE, int PROJ, int TL = G::LOG2L>
__global__ void __launch_bounds__(G::T, RGeom<G>::MINB_COL) col_pass_rk(ColArgs a) {
  constexpr int N = G::N, L = G::L, T = G::T;
  static_assert(TL == G::LOG2L || MODE == COL_FFT, "the iteration's tiles are as wide as its CTAs");
  using F0 = RFirst<G, 0>;
  using FL = RLast<G, 0>;   // == RFirst<G, 1> in shape
  using IL = RLast<G, 1>;
  static_assert(FL::R == RFirst<G, 1>::R && FL::B == RFirst<G, 1>::B, "plan 1 starts where plan 0 ends");
  extern __shared__ float2 smem[];
  __shared__ double red[T / 32];
  const float2* __restrict__ tw = a.tw;
  float2* buf = smem;
  const int c0 = blockIdx.x * L;
  const int ncols = min(L, a.cols - c0);
  const long long C = a.cols;
  const long long tile = (long long)blockIdx.x * N * L;

  constexpr bool iter = MODE == COL_ITER;
  float* amp_s = reinterpret_cast<float*>(smem + L * G::LD);
  float* int_s = amp_s + L * N;
  float* bs_s = int_s + L * N;
  const long long aux = (long long)blockIdx.y * a.aux_stride + tile;
  // the tile's sqrt(I) (and I, beamstop for PROJ_CCD): contiguous runs of L*N
  // floats, one bulk copy each, landing during the forward transform.  They start
  // before the wait for the row pass unless launches of the same call wrote the arrays
  // (a.aux_late): a context's patterns were complete when the host enqueued the run.
  // Frozen patterns copy nothing (a.may_stop): the flag as it stands ahead of the wait says
  // whether to start early, the flag after it what is done.  Us per iteration of a batch
  // whose patterns have all stopped, staging first and so: 2048^2 x4 32.8 -> 22.7, 256^2 x1024
  // 116 -> 92, 512^2 x48 with CCD noise and a beamstop 38.8 -> 22.1; running, 1 % or less either way.
  __shared__ uint64_t stage_bar;
  if constexpr (iter && bulk_staging<N>()) {
    if (threadIdx.x == 0) bulk_bar_init(&stage_bar);
    __syncthreads();
  }
  auto stage = [&]() {
    if constexpr (bulk_staging<N>()) {
      constexpr unsigned bytes = L * N * (unsigned)sizeof(float);
      if (threadIdx.x == 0) {
        const bool two = PROJ == PROJ_CCD, three = PROJ == PROJ_CCD && a.bs != nullptr;
        bulk_expect(&stage_bar, bytes * (1u + (two ? 1u : 0u) + (three ? 1u : 0u)));
        bulk_g2s(amp_s, a.amp + aux, bytes, &stage_bar);
        if (two) bulk_g2s(int_s, a.inten + aux, bytes, &stage_bar);
        if (three) bulk_g2s(bs_s, a.bs + aux, bytes, &stage_bar);
      }
    } else {
#pragma unroll 4
      for (int q = threadIdx.x; q < L * N / 4; q += T) {
        cp_async16(amp_s + 4 * q, a.amp + aux + 4 * q, true);
        if constexpr (PROJ == PROJ_CCD) {
          cp_async16(int_s + 4 * q, a.inten + aux + 4 * q, true);
          if (a.bs) cp_async16(bs_s + 4 * q, a.bs + aux + 4 * q, true);
        }
      }
      cp_commit();
    }
  };
  const bool early = iter && !a.aux_late && !(a.may_stop && (__ldcg(&a.state[blockIdx.y].flags) & 6));
#pragma unroll 1
  for (int waited = 0; waited < 2; ++waited) {   // one copy of the staging code: a second costs registers (192: 63 -> 69)
    if (waited) {
      pdl_wait_and_release();
      if (a.state) {
        const int f = a.state[blockIdx.y].flags;
        if (f & 6) {
          if ((f & 4) == 0 && threadIdx.x == 0) atomicOr(&a.state[blockIdx.y].flags, 4);
          if constexpr (iter) if (early) {   // a thread's copies land before it ends
            if constexpr (bulk_staging<N>()) { if (threadIdx.x == 0) bulk_wait(&stage_bar, a.err); }
            else cp_wait<0>();
          }
          return;
        }
      }
    }
    if constexpr (iter) if (waited != (int)early) stage();
  }
  const float2* in = a.in + (long long)blockIdx.y * a.in_stride;
  const bool in_t = a.in_tiled != 0;
  auto gload = [&](int l, int m) -> float2 {
    if constexpr (TL == G::LOG2L) {
      if (in_t) return __ldcg(in + tile + (long long)m * L + l);
    } else {
      if (in_t && l < ncols)   // tile (c0 + l) >> TL of the CTA's columns
        return __ldcg(in + tile + (long long)(l >> TL) * (N << TL) + (m << TL) + (l & ((1 << TL) - 1)));
    }
    return l < ncols ? __ldcg(in + m * C + c0 + l) : make_float2(0.f, 0.f);
  };
  float2 v[FL::B][FL::R];
  const bool fwd_fft = !iter || !a.from_psi;
  if (fwd_fft) {
    float2 v0[F0::B][F0::R];
#pragma unroll
    for (int b = 0; b < F0::B; ++b) {
      int l, j;
      if (!bfly_of<G, F0::R>(b, 0, l, j)) continue;
#pragma unroll
      for (int r = 0; r < F0::R; ++r) v0[b][r] = gload(l, j + r * F0::NR);
    }
    if (!iter && a.inv) rfft<G, 0, true>(v0, v, buf, tw, 0);
    else rfft<G, 0, false>(v0, v, buf, tw, 0);
  } else {
    // Psi given: load it where the forward transform would have left it
#pragma unroll
    for (int b = 0; b < FL::B; ++b) {
      int l, j;
      if (!bfly_of<G, FL::R>(b, 0, l, j)) continue;
#pragma unroll
      for (int r = 0; r < FL::R; ++r) v[b][r] = gload(l, j + r * FL::NS);
    }
  }
  float2* out = a.out + (long long)blockIdx.y * a.out_stride;
  const bool out_t = a.out_tiled != 0;
  const float s = a.scale;
  if constexpr (!iter) {
#pragma unroll
    for (int b = 0; b < FL::B; ++b) {
      int l, j;
      if (!bfly_of<G, FL::R>(b, 0, l, j)) continue;
#pragma unroll
      for (int r = 0; r < FL::R; ++r) {
        const int m = j + r * FL::NS;
        float2 y = v[b][r];
        if (s != 1.f) { y.x *= s; y.y *= s; }
        if (TL == G::LOG2L && out_t) __stcg(out + tile + (long long)m * L + l, y);
        else if (l < ncols) __stcg(out + m * C + c0 + l, y);
      }
    }
    return;
  } else {
    if constexpr (bulk_staging<N>()) bulk_wait(&stage_bar, a.err);
    else cp_wait<0>();
    __syncthreads();
    // Psi complete in registers: optional R-factor partial (one loop behind
    // one uniform branch), then the projection (branch-free per element, so
    // the compiler interleaves the elements), then the optional copy-out of P_M Psi
    if (a.rf_partials) {
      double rsum = 0.0;
#pragma unroll
      for (int b = 0; b < FL::B; ++b) {
        int l, j;
        if (!bfly_of<G, FL::R>(b, 0, l, j) || l >= ncols) continue;
#pragma unroll
        for (int r = 0; r < FL::R; ++r) {
          const float2 z = v[b][r];
          rsum += fabsf(hypotf(z.x, z.y) - amp_s[(j + r * FL::NS) * L + l]);
        }
      }
      const double tsum = block_sum_d<T>(rsum, red);
      if (threadIdx.x == 0) a.rf_partials[(long long)blockIdx.y * gridDim.x + blockIdx.x] = tsum;
    }
#pragma unroll
    for (int b = 0; b < FL::B; ++b) {
      int l, j;
      if (!bfly_of<G, FL::R>(b, 0, l, j)) continue;
#pragma unroll
      for (int r = 0; r < FL::R; ++r) {
        const int t = (j + r * FL::NS) * L + l;
        float2 z = v[b][r];
        if constexpr (PROJ == PROJ_MODABS) z = proj_modabs(z, amp_s[t]);
        else z = proj_ccd(z, int_s[t], a.bs ? bs_s[t] : 0.f, a.bs != nullptr, a.noise_level, a.ccd_scale,
                          a.ccd_rcolor);
        v[b][r] = l < ncols ? z : make_float2(0.f, 0.f);
      }
    }
    if (a.psi_out) {
      float2* psi_out = a.psi_out + (long long)blockIdx.y * a.psi_stride;
#pragma unroll
      for (int b = 0; b < FL::B; ++b) {
        int l, j;
        if (!bfly_of<G, FL::R>(b, 0, l, j) || l >= ncols) continue;
#pragma unroll
        for (int r = 0; r < FL::R; ++r) psi_out[(j + r * FL::NS) * C + c0 + l] = v[b][r];
      }
    }
    float2 o[IL::B][IL::R];
    rfft<G, 1, true>(v, o, buf, tw, 0);
#pragma unroll
    for (int b = 0; b < IL::B; ++b) {
      int l, j;
      if (!bfly_of<G, IL::R>(b, 0, l, j)) continue;
#pragma unroll
      for (int r = 0; r < IL::R; ++r) {
        const int m = j + r * IL::NS;
        float2 y = o[b][r];
        if (s != 1.f) { y.x *= s; y.y *= s; }
        if (out_t) __stcg(out + tile + (long long)m * L + l, y);
        else if (l < ncols) __stcg(out + m * C + c0 + l, y);
      }
    }
  }
}

// ------------------------------------------------------------------- row pass
// Lines are rows (length N = cols).  Column-tiled arrays have tile width
// 2^tile_log2 (the column pass's L for the row count).
// SQ (ROW_ITER only): W is column-tiled on both sides with the tile width of a
// column pass of length N (square patterns) and the butterflies use the default
// chunk, so the layout is known at compile time: each butterfly's 16 elements
// are one base address plus whole-tile strides, with no per-element index
// arithmetic.  The launcher takes the general kernel otherwise.
// The compile-time layout needs every pass's element stride to be whole tiles:
// 2^log2(L) divides N/R for each radix R (true from 128 up, and from 256 up with the
// wider tiles of Geom; below, the column tiles are wider than that).
template <class G>
__host__ __device__ constexpr bool row_sq_ok_g() { return G::LOG2L <= rfft_cb_max<G::N>(); }
template <int N>
__host__ __device__ constexpr bool row_sq_ok() { return row_sq_ok_g<Geom<N>>(); }

template <class G, int MODE, int ALGO, bool SQ = false>
__device__ __forceinline__ void row_pass_body(const RowArgs& a) {
  constexpr int N = G::N, L = G::L, T = G::T, LD = RGeom<G>::ROW_LD;
  using F0 = RFirst<G, 0>;
  using FL = RLast<G, 0>;
  using IL = RLast<G, 1>;
  static_assert(FL::R == RFirst<G, 1>::R && FL::B == RFirst<G, 1>::B, "plan 1 starts where plan 0 ends");
  extern __shared__ float2 smem[];
  const float2* __restrict__ tw = a.tw;
  float2* buf = smem;
  const int row0 = blockIdx.x * L;
  const int nrows = min(L, a.rows - row0);
  constexpr bool iter = MODE == ROW_ITER;
  constexpr bool CT = SQ && iter && row_sq_ok_g<G>();   // compile-time layout
  constexpr int TLC = G::LOG2L;
  constexpr int CBC = row_cb_pick(TLC, rfft_cb_max<N>());
  const int tl = CT ? TLC : a.tile_log2;
  // tiled: four (or 2^tl) threads per tile row piece; row-major: consecutive
  // threads take consecutive columns
  const bool tiled = a.in_tiled || a.out_tiled;
  const int cb = CT ? CBC
                    : (a.cb_plus1 > 0 ? min(a.cb_plus1 - 1, rfft_cb_max<N>())
                                      : (tiled ? row_cb_pick(tl, rfft_cb_max<N>()) : rfft_cb_max<N>()));

  // rho rows and support words of the CTA (ROW_ITER), landing during the inverse FFT
  // (RHO_IN_BUF: the rho rows land in the line buffer during its last pass)
  constexpr int RS = LD;                    // rho line stride in shared memory
  constexpr int WPR = (N + 31) >> 5;
  // Support words in shared memory: with MT the words a butterfly of the update
  // needs (columns j + r*NS, r < R: word (j >> 5) + r*NS/32) are staged next to
  // one another, so a thread reads its R words with R/4 16-byte loads instead of R.
  constexpr bool MT = FL::NS % 32 == 0 && FL::R % 4 == 0 && WPR % 4 == 0;
  constexpr int MG = MT ? FL::NS / 32 : 1;   // word groups per row
  auto mask_slot = [](int w) -> int {
    if constexpr (MT) {
      const int l = w / WPR, q = w - l * WPR;   // row l, word q = g + r*MG
      return l * WPR + (q % MG) * FL::R + q / MG;
    } else {
      return w;
    }
  };
  constexpr bool rho_in_buf = RGeom<G>::RHO_IN_BUF;
  float2* rho_s = rho_in_buf ? smem : smem + L * LD;
  uint32_t* mask_s = reinterpret_cast<uint32_t*>(smem + L * LD + (rho_in_buf ? 0 : L * RS));
  float2* rho = a.rho + (long long)blockIdx.y * a.rho_stride + (long long)row0 * N;
  // with an even line stride each rho row is one bulk copy (16-byte aligned); from 32 rows
  // per CTA on, one thread issuing them is slower than 16-byte pieces by all (64^2: 14.4 -> 12.9 us)
  constexpr bool bulk_rho = bulk_staging<N>() && RS % 2 == 0 && L <= 16;
  __shared__ uint64_t rho_bar;
  if constexpr (iter && bulk_rho) {
    if (threadIdx.x == 0) bulk_bar_init(&rho_bar);
    __syncthreads();
  }
  // the rho rows: one bulk copy per row, or 16- / 8-byte cp.async pieces
  auto stage_rho = [&]() {
    if constexpr (bulk_rho) {
      if (threadIdx.x == 0) {
        // the lines were last read through the generic proxy: order that before the bulk writes
        if constexpr (rho_in_buf) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        bulk_expect(&rho_bar, (unsigned)nrows * N * (unsigned)sizeof(float2));
        for (int l = 0; l < nrows; ++l)
          bulk_g2s(rho_s + l * RS, rho + (long long)l * N, N * (unsigned)sizeof(float2), &rho_bar);
      }
    } else if constexpr (RS % 2 == 0) {
#pragma unroll 4
      for (int e = threadIdx.x; e < L * N / 2; e += T) {
        const int l = (2 * e) / N, c = 2 * e - l * N;
        const bool ok = l < nrows;
        cp_async16(rho_s + l * RS + c, ok ? rho + 2 * e : rho, ok);
      }
    } else {
#pragma unroll 4
      for (int e = threadIdx.x; e < L * N; e += T) {
        const int l = e / N, c = e - l * N;
        const bool ok = l < nrows;
        cp_async8(rho_s + l * RS + c, ok ? rho + e : rho, ok);
      }
    }
  };
  // rho and the support words are the run's own data: no value of them is read before the
  // wait.  Rows copied in late start towards L2 ahead of it, but not those of a frozen pattern.
  if constexpr (iter && rho_in_buf)
    if (threadIdx.x < nrows && !(a.may_stop && (__ldcg(&a.state[blockIdx.y].flags) & 4)))
      bulk_prefetch_l2(rho + (long long)threadIdx.x * N, N * (unsigned)sizeof(float2));
  pdl_wait_and_release();
  if (a.state && (a.state[blockIdx.y].flags & 4)) return;   // frozen pattern
  const float2* in = a.in + (long long)blockIdx.y * a.in_stride;
  const long long R = a.rows;
  auto goff = [&](bool t, int l, int c) -> long long {
    const int row = row0 + l;
    return t ? ((((long long)(c >> tl)) * R + row) << tl) + (c & ((1 << tl) - 1)) : (long long)row * N + c;
  };
  float2 v[FL::B][FL::R];
  {
    float2 v0[F0::B][F0::R];
#pragma unroll
    for (int b = 0; b < F0::B; ++b) {
      int l, j;
      if (!bfly_of<G, F0::R>(b, cb, l, j)) continue;
      if constexpr (CT) {
        // element j + r*NR: tile (j >> TLC) + r*(NR >> TLC), lane j & (2^TLC - 1)
        static_assert(F0::NR % (1 << TLC) == 0, "first-pass stride is whole tiles");
        const float2* p = in + ((((long long)(j >> TLC)) * R + row0 + l) << TLC) + (j & ((1 << TLC) - 1));
        const long long st = ((long long)(F0::NR >> TLC) * R) << TLC;
#pragma unroll
        for (int r = 0; r < F0::R; ++r) v0[b][r] = l < nrows ? __ldcg(p + r * st) : make_float2(0.f, 0.f);
      } else {
#pragma unroll
        for (int r = 0; r < F0::R; ++r)
          v0[b][r] = l < nrows ? __ldcg(in + goff(a.in_tiled, l, j + r * F0::NR)) : make_float2(0.f, 0.f);
      }
    }
    if constexpr (iter) {   // behind the loads of W
      if constexpr (!rho_in_buf) stage_rho();
      const uint32_t* mask = a.mask + (long long)blockIdx.y * a.mask_stride + (long long)row0 * WPR;
      for (int w = threadIdx.x; w < L * WPR; w += T) {
        const bool ok = w / WPR < nrows;
        cp_async4(mask_s + mask_slot(w), ok ? mask + w : mask, ok);
      }
      cp_commit();
    }
    if constexpr (iter && rho_in_buf) {
      rfft<G, 0, true, LD>(v0, v, buf, tw, cb, [&]() {
        __syncthreads();   // every thread's last read of the lines is done
        stage_rho();
        cp_commit();
      });
    } else if (iter || a.inv) {
      rfft<G, 0, true, LD>(v0, v, buf, tw, cb);
    } else {
      rfft<G, 0, false, LD>(v0, v, buf, tw, cb);
    }
  }
  float2* out = a.out + (long long)blockIdx.y * a.out_stride;
  const float s = a.scale;
  if constexpr (!iter) {
#pragma unroll
    for (int b = 0; b < FL::B; ++b) {
      int l, j;
      if (!bfly_of<G, FL::R>(b, cb, l, j)) continue;
      if (l >= nrows) continue;
#pragma unroll
      for (int r = 0; r < FL::R; ++r) {
        float2 y = v[b][r];
        if (s != 1.f) { y.x *= s; y.y *= s; }
        __stcg(out + goff(a.out_tiled, l, j + r * FL::NS), y);
      }
    }
  } else {
    cp_wait<0>();
    if constexpr (bulk_rho) bulk_wait(&rho_bar, a.err);
    __syncthreads();
    // rho' = IFFT/N; update against rho and the support bits
#pragma unroll
    for (int b = 0; b < FL::B; ++b) {
      int l, j;
      if (!bfly_of<G, FL::R>(b, cb, l, j)) continue;
      const uint4* m4 = reinterpret_cast<const uint4*>(mask_s + l * WPR + (j >> 5) * FL::R);
      uint4 mq = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int r = 0; r < FL::R; ++r) {
        const int c = j + r * FL::NS;
        float2 y = make_float2(0.f, 0.f);
        if constexpr (MT) if ((r & 3) == 0) mq = m4[r >> 2];   // four words at a time
        if (l < nrows) {
          float2 p = v[b][r];
          p.x *= a.inv_n;
          p.y *= a.inv_n;
          const float2 x = rho_s[l * RS + c];
          const uint32_t word = MT ? ((r & 3) == 0 ? mq.x : (r & 3) == 1 ? mq.y : (r & 3) == 2 ? mq.z : mq.w)
                                   : mask_s[l * WPR + (c >> 5)];
          const bool inside = (word >> (c & 31)) & 1u;
          y = update_t<ALGO>(inside, x, p, a.beta);
          rho[l * N + c] = y;
        }
        v[b][r] = y;
      }
    }
    float2 o[IL::B][IL::R];
    if constexpr (rho_in_buf) __syncthreads();   // the rho rows are read before the lines are reused
    rfft<G, 1, false, LD>(v, o, buf, tw, cb);
#pragma unroll
    for (int b = 0; b < IL::B; ++b) {
      int l, j;
      if (!bfly_of<G, IL::R>(b, cb, l, j)) continue;
      if (l >= nrows) continue;
      if constexpr (CT) {
        static_assert(IL::NS % (1 << TLC) == 0, "last-pass stride is whole tiles");
        float2* p = out + ((((long long)(j >> TLC)) * R + row0 + l) << TLC) + (j & ((1 << TLC) - 1));
        const long long st = ((long long)(IL::NS >> TLC) * R) << TLC;
#pragma unroll
        for (int r = 0; r < IL::R; ++r) __stcg(p + r * st, o[b][r]);   // the iteration stores unscaled
      } else {
#pragma unroll
        for (int r = 0; r < IL::R; ++r) {
          float2 y = o[b][r];
          if (s != 1.f) { y.x *= s; y.y *= s; }
          __stcg(out + goff(a.out_tiled, l, j + r * IL::NS), y);
        }
      }
    }
  }
}

// One kernel per update (ALGO is ignored in ROW_FFT mode): the executed code
// holds a single update and no switch.
template <class G, int MODE, int ALGO, bool SQ = false>
__global__ void __launch_bounds__(G::T, MODE == ROW_FFT ? RGeom<G>::MINB_ROW_FFT : RGeom<G>::MINB_ROW) row_pass_rk(RowArgs a) {
  row_pass_body<G, MODE, ALGO, SQ>(a);
}
// the compile-time layout of row_pass_rk<..., true> applies to these arguments
template <class G>
__host__ __forceinline__ bool row_sq_layout(const RowArgs& a) {
  constexpr int cbd = row_cb_pick(G::LOG2L, rfft_cb_max<G::N>());
  return row_sq_ok_g<G>() && a.mode == ROW_ITER && a.in_tiled && a.out_tiled && a.tile_log2 == G::LOG2L && a.scale == 1.f &&
         (a.cb_plus1 == 0 || a.cb_plus1 - 1 == cbd);
}

}  // namespace cdx
