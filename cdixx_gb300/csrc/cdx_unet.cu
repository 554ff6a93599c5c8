// Warm-start U-Net: layer graph, element-wise kernels (GroupNorm, LeakyReLU,
// loss, Adam) and the C ABI of include/cdx_unet.h.  The convolutions are the
// implicit-GEMM tensor-core kernels of cdx_unet_gemm.cuh.
//
// Flat parameter order (FP32): layers in forward order; per layer the weight
// (conv layout [Cout][KH][KW][Cin]; a transposed convolution stores the
// convolution it is the adjoint of, [Cin_T][2][2][Cout_T]), then GroupNorm
// gamma[C] and beta[C]; the head has weight [4][1][1][base] and bias[4].
// The first convolution sees one input channel.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>
#include <cstring>
#include <string>
#include <vector>

#include "cdx.h"
#include "cdx_host.h"
#include "cdx_types.h"
#include "cdx_unet.h"
#include "cdx_unet_gemm.cuh"
#include "cdx_unet_umma.cuh"

namespace cdx {
namespace unet {

#define U_CK(call)                                                                                \
  do {                                                                                            \
    cudaError_t e_ = (call);                                                                      \
    if (e_ != cudaSuccess) return set_error(CDX_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

constexpr int kThreads = 256;

// ------------------------------------------------------------ element-wise kernels
// The largest log(1 + I) of each pattern, as float bits (values are >= 0, so
// unsigned order is float order): one slice of a pattern per CTA, so that a few
// patterns still use every SM (one CTA per pattern took 174 us for 8 of 256^2).
__global__ void k_prep_max(const float* __restrict__ inten, int P, unsigned* __restrict__ mx) {
  const float* I = inten + (long long)blockIdx.x * P;
  float m = 0.f;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < P; i += gridDim.y * blockDim.x)
    m = fmaxf(m, log1pf(fmaxf(I[i], 0.f)));
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(mx + blockIdx.x, __float_as_uint(m));
}
// log(1 + I) / max log(1 + I) per pattern, centred (fftshift), channel 0 of 8 (one 16-byte store)
__global__ void k_prep_input(const float* __restrict__ inten, const unsigned* __restrict__ mx,
                             __nv_bfloat16* __restrict__ x, int n) {
  net_wait();
  const int P = n * n, h = n / 2;
  const float* I = inten + (long long)blockIdx.x * P;
  const float top = __uint_as_float(mx[blockIdx.x]);
  const float inv = top > 0.f ? 1.f / top : 0.f;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < P; i += gridDim.y * blockDim.x) {
    const int y = i / n, xx = i - y * n;
    const int sy = y < h ? y + h : y - h, sx = xx < h ? xx + h : xx - h;   // centred pixel <- FFT-order pixel
    const float v = log1pf(fmaxf(I[sy * n + sx], 0.f)) * inv;
    const __nv_bfloat162 b = __halves2bfloat162(__float2bfloat16(v), __float2bfloat16(0.f));
    reinterpret_cast<uint4*>(x)[(long long)blockIdx.x * P + i] =
        make_uint4(*reinterpret_cast<const unsigned*>(&b), 0u, 0u, 0u);
  }
}

// FP32 weights [co][kh][kw][ci] (real sizes) -> BF16 [co_p][kh][kw][ci_p] and
// transposed [ci_p][kh][kw][co_p], zero-padded, and both packed for k_conv_umma
// ([K/8][columns][8], K = (kh, kw, ci) or (kh, kw, co))
__global__ void k_weights_bf16(const float* __restrict__ w, int co_r, int ci_r, int co_p, int ci_p, int kk,
                               __nv_bfloat16* __restrict__ wb, __nv_bfloat16* __restrict__ wt,
                               __nv_bfloat16* __restrict__ pb, __nv_bfloat16* __restrict__ pt) {
  const long long total = (long long)co_p * kk * ci_p;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int ci = (int)(i % ci_p);
    const long long t = i / ci_p;
    const int k = (int)(t % kk), co = (int)(t / kk);
    const float v = (co < co_r && ci < ci_r) ? w[((long long)co * kk + k) * ci_r + ci] : 0.f;
    const __nv_bfloat16 b = __float2bfloat16(v);
    wb[i] = b;
    wt[((long long)ci * kk + k) * co_p + co] = b;
    const int kb = k * ci_p + ci, kt = k * co_p + co;
    pb[((long long)(kb >> 3) * co_p + co) * 8 + (kb & 7)] = b;
    pt[((long long)(kt >> 3) * ci_p + ci) * 8 + (kt & 7)] = b;
  }
}

// sum of wgrad partials over the splits, cropped to the real weight shape
__global__ void k_wgrad_reduce(const float* __restrict__ part, int splits, int co_r, int ci_r, int co_p, int ci_p,
                               int kk, float* __restrict__ grad) {
  const long long total = (long long)co_r * kk * ci_r;
  const long long stride = (long long)co_p * kk * ci_p;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int ci = (int)(i % ci_r);
    const long long t = i / ci_r;
    const int k = (int)(t % kk), co = (int)(t / kk);
    const long long src = ((long long)co * kk + k) * ci_p + ci;
    float s = 0.f;
    for (int z = 0; z < splits; ++z) s += part[z * stride + src];
    grad[i] = s;
  }
}

// ---- GroupNorm + LeakyReLU.  All of it is bound by HBM, so every kernel reads
// 16-byte pieces, several in flight per thread.  The statistics keep one running
// float sum per channel and pixel class (pixel mod 256 / Cg within the split) and
// fold them in double in a fixed tree: a CTA takes gpc groups, whole 128-byte
// lines of channels where they allow it, a thread four channels of one class.
// b = 32 at 256^2, per training step: statistics 611 -> 443 us, apply 2067 -> 509,
// backward statistics 1658 -> 916, backward apply 2240 -> 936 (8 channels a CTA:
// 486 and 976; loads not batched: 1286 and 1168).
inline int gn_groups(int Cg, int G) {   // groups per CTA: up to 32 channels, a power of two that divides G
  int g = 1;
  while (g < 8 && Cg * g < 32 && G % (2 * g) == 0) g *= 2;
  return g;
}

// fixed tree over the 256 class sums of each of `gpc` groups in r (256 doubles per group), down to `stop` sums
__device__ __forceinline__ void gn_tree(double* r, int gpc, int stop) {
  __syncthreads();
  for (int o = kThreads / 2; o >= stop; o >>= 1) {
    for (int i = threadIdx.x; i < gpc * o; i += blockDim.x) {
      const int gl = i / o, k = i - gl * o;
      r[gl * kThreads + k] += r[gl * kThreads + k + o];
    }
    __syncthreads();
  }
}

// statistics: partial sums per (pattern, group, split); grid (patterns, split, G / gpc)
__global__ void __launch_bounds__(512) k_gn_stats(const float* __restrict__ x, int HW, int C, int G, int gpc,
                                                  int split, double* __restrict__ part) {
  net_wait();
  const int n = blockIdx.x, z = blockIdx.y, Cg = C / G, kc = gpc * Cg, tpc = kThreads / Cg;
  const int q4 = kc / 4, q = threadIdx.x % q4, p0 = threadIdx.x / q4;
  const int pb = (int)((long long)HW * z / split), pe = (int)((long long)HW * (z + 1) / split);
  const float4* base = reinterpret_cast<const float4*>(x + (long long)n * HW * C + blockIdx.z * kc) + q;
  const int C4 = C / 4;
  float s[4] = {0.f, 0.f, 0.f, 0.f}, ss[4] = {0.f, 0.f, 0.f, 0.f};
  auto add = [&](const float4& f) {
    const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      s[k] += v[k];
      ss[k] += v[k] * v[k];
    }
  };
  // batches of eight loads, the next batch in flight while this one is added
  constexpr int U = 8;
  float4 f[U], g[U];
  int p = pb + p0;
  const int nb = p < pe ? ((pe - 1 - p) / tpc + 1) / U : 0;   // whole batches
  const long long st = (long long)tpc * C4;
  const float4* b = base + (long long)p * C4;
  if (nb > 0) {
#pragma unroll
    for (int u = 0; u < U; ++u) f[u] = __ldg(b + u * st);
  }
  for (int i = 0; i < nb; ++i) {
    b += U * st;
    if (i + 1 < nb) {
#pragma unroll
      for (int u = 0; u < U; ++u) g[u] = __ldg(b + u * st);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) add(f[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) f[u] = g[u];
  }
  for (p += nb * U * tpc; p < pe; p += tpc, b += st) add(__ldg(b));
  extern __shared__ double r[];   // gpc x 256, classes of one group: class * Cg + channel
  const int g0 = blockIdx.z * gpc;
  for (int what = 0; what < 2; ++what) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * q + k;
      r[c / Cg * kThreads + p0 * Cg + c % Cg] = what ? ss[k] : s[k];
    }
    gn_tree(r, gpc, 1);
    if (threadIdx.x < gpc) part[(((long long)n * G + g0 + threadIdx.x) * split + z) * 2 + what] = r[threadIdx.x * kThreads];
  }
}

// Element-wise GroupNorm kernels: a CTA takes a range of pixels (grid.y) of one pattern
// (grid.x) and, a thread each, eight channels of a pixel; octets beyond 256 go to
// grid.z.  A thread keeps its channels over the range, so the per-channel values
// stay in registers.
struct GnSpan {
  int oct, p, pe, step;
  bool ok;
};
__host__ __device__ constexpr int gn_octs(int C) { return C / 8 < kThreads ? C / 8 : kThreads; }
__device__ __forceinline__ GnSpan gn_span(int HW, int C) {
  GnSpan s;
  const int oc = gn_octs(C);
  s.step = kThreads / oc;
  s.oct = blockIdx.z * oc + threadIdx.x % oc;
  const int r = threadIdx.x / oc;
  s.ok = r < s.step && s.oct < C / 8;
  s.p = (int)((long long)HW * blockIdx.y / gridDim.y) + r;
  s.pe = (int)((long long)HW * (blockIdx.y + 1) / gridDim.y);
  return s;
}
__device__ __forceinline__ void ld8(float (&v)[8], const float* p) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void st8(__nv_bfloat16* p, const float (&v)[8]) {
  __nv_bfloat162 h[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) h[k] = __halves2bfloat162(__float2bfloat16(v[2 * k]), __float2bfloat16(v[2 * k + 1]));
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(h);
}

// y = LeakyReLU(gamma (x - mean) rstd + beta) -> BF16.  The statistics are
// finished here: every CTA folds its pattern's `split` partials (a few hundred
// bytes) in order, and the first one of a pattern keeps mean and rstd for the backward.
__global__ void __launch_bounds__(kThreads) k_gn_apply(const float* __restrict__ x, const double* __restrict__ part,
                                                       int split, float* __restrict__ stats,
                                                       const float* __restrict__ gamma, const float* __restrict__ beta,
                                                       int HW, int C, int G, float slope, __nv_bfloat16* __restrict__ y) {
  extern __shared__ float2 st[];   // mean, rstd per group
  net_wait();
  const int n = blockIdx.x, Cg = C / G;
  for (int g = threadIdx.x; g < G; g += kThreads) {
    double s = 0.0, q = 0.0;
#pragma unroll 8
    for (int z = 0; z < split; ++z) {
      const double2 v = reinterpret_cast<const double2*>(part)[((long long)n * G + g) * split + z];
      s += v.x;
      q += v.y;
    }
    const double count = (double)HW * Cg;
    const double mean = s / count;
    const double var = fmax(q / count - mean * mean, 0.0);
    st[g] = make_float2((float)mean, (float)(1.0 / sqrt(var + 1e-5)));
    if (blockIdx.y == 0 && blockIdx.z == 0) reinterpret_cast<float2*>(stats)[n * G + g] = st[g];
  }
  __syncthreads();
  const GnSpan t = gn_span(HW, C);
  if (!t.ok) return;
  const int c0 = t.oct * 8;
  float ga[8], be[8], mean[8], rstd[8];
  ld8(ga, gamma + c0);
  ld8(be, beta + c0);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float2 v = st[(c0 + k) / Cg];
    mean[k] = v.x;
    rstd[k] = v.y;
  }
  const long long off = (long long)n * HW * C + c0;
#pragma unroll 4
  for (int p = t.p; p < t.pe; p += t.step) {
    float v[8];
    ld8(v, x + off + (long long)p * C);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float z = (v[k] - mean[k]) * rstd[k] * ga[k] + be[k];
      v[k] = z > 0.f ? z : slope * z;
    }
    st8(y + off + (long long)p * C, v);
  }
}

// backward, pass 1: per (pattern, group, split) sums of dz*gamma and
// dz*gamma*xhat, per channel sums of dz*xhat and dz; grid as k_gn_stats
__global__ void __launch_bounds__(512) k_gn_bwd_stats(const float* __restrict__ x, const float* __restrict__ dy,
                                                      const float* __restrict__ stats, const float* __restrict__ gamma,
                                                      const float* __restrict__ beta, int HW, int C, int G, int gpc,
                                                      int split, float slope, double* __restrict__ part_g,
                                                      double* __restrict__ part_c) {
  const int n = blockIdx.x, z = blockIdx.y, Cg = C / G, kc = gpc * Cg, tpc = kThreads / Cg;
  const int q4 = kc / 4, q = threadIdx.x % q4, p0 = threadIdx.x / q4;
  const int g0 = blockIdx.z * gpc, ch0 = blockIdx.z * kc;
  const int pb = (int)((long long)HW * z / split), pe = (int)((long long)HW * (z + 1) / split);
  float mean[4], rstd[4], ga[4], be[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = ch0 + 4 * q + k;
    const long long ng = (long long)n * G + c / Cg;
    mean[k] = stats[2 * ng];
    rstd[k] = stats[2 * ng + 1];
    ga[k] = gamma[c];
    be[k] = beta[c];
  }
  const long long off = ((long long)n * HW * C + ch0) / 4 + q;
  const float4* xb = reinterpret_cast<const float4*>(x) + off;
  const float4* db4 = reinterpret_cast<const float4*>(dy) + off;
  const int C4 = C / 4;
  float s1[4] = {}, s2[4] = {}, dg[4] = {}, db[4] = {};
  auto add = [&](const float4& fx, const float4& fd) {
    const float vx[4] = {fx.x, fx.y, fx.z, fx.w}, vd[4] = {fd.x, fd.y, fd.z, fd.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float xh = (vx[k] - mean[k]) * rstd[k];
      const float zz = xh * ga[k] + be[k];
      const float dz = vd[k] * (zz > 0.f ? 1.f : slope);
      s1[k] += dz * ga[k];
      s2[k] += dz * ga[k] * xh;
      dg[k] += dz * xh;
      db[k] += dz;
    }
  };
  constexpr int U = 4;   // batches as in k_gn_stats
  float4 f[2][U], g[2][U];
  int p = pb + p0;
  const int nb = p < pe ? ((pe - 1 - p) / tpc + 1) / U : 0;
  const long long st = (long long)tpc * C4;
  xb += (long long)p * C4;
  db4 += (long long)p * C4;
  if (nb > 0) {
#pragma unroll
    for (int u = 0; u < U; ++u) { f[0][u] = __ldg(xb + u * st); f[1][u] = __ldg(db4 + u * st); }
  }
  for (int i = 0; i < nb; ++i) {
    xb += U * st;
    db4 += U * st;
    if (i + 1 < nb) {
#pragma unroll
      for (int u = 0; u < U; ++u) { g[0][u] = __ldg(xb + u * st); g[1][u] = __ldg(db4 + u * st); }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) add(f[0][u], f[1][u]);
#pragma unroll
    for (int u = 0; u < U; ++u) { f[0][u] = g[0][u]; f[1][u] = g[1][u]; }
  }
  for (p += nb * U * tpc; p < pe; p += tpc, xb += st, db4 += st) add(__ldg(xb), __ldg(db4));
  extern __shared__ double r[];
  for (int what = 0; what < 4; ++what) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = 4 * q + k;
      r[c / Cg * kThreads + p0 * Cg + c % Cg] = what == 0 ? s1[k] : what == 1 ? s2[k] : what == 2 ? dg[k] : db[k];
    }
    gn_tree(r, gpc, Cg);   // Cg channel sums per group
    if (what < 2) {
      if (threadIdx.x < gpc) {
        double a = 0.0;
        for (int k = 0; k < Cg; ++k) a += r[threadIdx.x * kThreads + k];
        part_g[(((long long)n * G + g0 + threadIdx.x) * split + z) * 2 + what] = a;
      }
    } else {
      for (int c = threadIdx.x; c < kc; c += blockDim.x)
        part_c[(((long long)n * split + z) * C + ch0 + c) * 2 + (what - 2)] = r[c / Cg * kThreads + c % Cg];
    }
  }
}

// pass 2: the gamma / beta gradients, one warp per channel over the patterns and splits (fixed order)
__global__ void k_gn_bwd_finalize(const double* __restrict__ part_c, int rows, int C, float* __restrict__ dgamma,
                                  float* __restrict__ dbeta) {
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= C) return;
  double a = 0.0, b = 0.0;
  for (int i = lane; i < rows; i += 32) {
    const double2 v = reinterpret_cast<const double2*>(part_c)[(long long)i * C + c];
    a += v.x;
    b += v.y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  if (lane == 0) {
    dgamma[c] = (float)a;
    dbeta[c] = (float)b;
  }
}

// pass 3: dx = rstd (dz gamma - S1/M - xhat S2/M) -> BF16; the group sums are
// folded here from the `split` partials, as in k_gn_apply
__global__ void __launch_bounds__(kThreads) k_gn_bwd_apply(const float* __restrict__ x, const float* __restrict__ dy,
                                                           const float* __restrict__ stats,
                                                           const double* __restrict__ part_g, int split,
                                                           const float* __restrict__ gamma, const float* __restrict__ beta,
                                                           int HW, int C, int G, float slope,
                                                           __nv_bfloat16* __restrict__ dx) {
  extern __shared__ float4 sg[];   // mean, rstd, S1, S2 per group
  const int n = blockIdx.x, Cg = C / G;
  const float inv_m = 1.f / ((float)HW * Cg);
  for (int g = threadIdx.x; g < G; g += kThreads) {
    const long long ng = (long long)n * G + g;
    double a = 0.0, b = 0.0;
#pragma unroll 8
    for (int z = 0; z < split; ++z) {
      const double2 v = reinterpret_cast<const double2*>(part_g)[ng * split + z];
      a += v.x;
      b += v.y;
    }
    sg[g] = make_float4(stats[2 * ng], stats[2 * ng + 1], (float)a, (float)b);
  }
  __syncthreads();
  const GnSpan t = gn_span(HW, C);
  if (!t.ok) return;
  const int c0 = t.oct * 8;
  float ga[8], be[8];
  ld8(ga, gamma + c0);
  ld8(be, beta + c0);
  const long long off = (long long)n * HW * C + c0;
#pragma unroll 2
  for (int p = t.p; p < t.pe; p += t.step) {
    float v[8], d[8];
    ld8(v, x + off + (long long)p * C);
    ld8(d, dy + off + (long long)p * C);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float4 s = sg[(c0 + k) / Cg];
      const float xh = (v[k] - s.x) * s.y;
      const float zz = xh * ga[k] + be[k];
      const float dz = d[k] * (zz > 0.f ? 1.f : slope);
      v[k] = s.y * (dz * ga[k] - s.z * inv_m - xh * s.w * inv_m);
    }
    st8(dx + off + (long long)p * C, v);
  }
}

// head bias: out[m][c] += bias[c], c < 4 (rows of 8 channels)
__global__ void k_bias_add(float* __restrict__ out, const float* __restrict__ bias, long long M) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < M * 4; i += (long long)gridDim.x * blockDim.x)
    out[(i >> 2) * 8 + (i & 3)] += bias[i & 3];
}

__device__ __forceinline__ float bce_logits(float z, float t) {
  return fmaxf(z, 0.f) - z * t + log1pf(expf(-fabsf(z)));
}
__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + expf(-z)); }

// per-pixel loss terms of the object (tw = 0) and its twin (tw = 1)
__device__ __forceinline__ float pixel_loss(const float* o, float at, float pt, float st, float ws) {
  float s, c;
  sincosf(pt, &s, &c);
  const float da = o[0] - at, dc = o[1] - c, ds = o[2] - s;
  return da * da + at * (dc * dc + ds * ds) + ws * bce_logits(o[3], st);
}

// partial loss sums per (pattern, split): [object, twin]
__global__ void k_loss_partial(const float* __restrict__ out, const float* __restrict__ amp_t,
                               const float* __restrict__ ph_t, const float* __restrict__ sup_t, int n, int split,
                               float ws, double* __restrict__ part) {
  const int b = blockIdx.x, z = blockIdx.y;
  const int P = n * n;
  const int pb = (int)((long long)P * z / split), pe = (int)((long long)P * (z + 1) / split);
  const long long o = (long long)b * P;
  float l0 = 0.f, l1 = 0.f;
  for (int p = pb + threadIdx.x; p < pe; p += blockDim.x) {
    const int y = p / n, x = p - y * n;
    const int q = ((n - y) % n) * n + (n - x) % n;   // twin pixel -r
    const float* op = out + (o + p) * 8;
    l0 += pixel_loss(op, amp_t[o + p], ph_t[o + p], sup_t[o + p], ws);
    l1 += pixel_loss(op, amp_t[o + q], -ph_t[o + q], sup_t[o + q], ws);
  }
  __shared__ double r0[kThreads], r1[kThreads];
  r0[threadIdx.x] = l0;
  r1[threadIdx.x] = l1;
  __syncthreads();
  for (int s = kThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      r0[threadIdx.x] += r0[threadIdx.x + s];
      r1[threadIdx.x] += r1[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[((long long)b * split + z) * 2] = r0[0];
    part[((long long)b * split + z) * 2 + 1] = r1[0];
  }
}

// per pattern (a thread each): the branch with the smaller loss; total = mean over patterns of the per-pixel mean
__global__ void k_loss_select(const double* __restrict__ part, int count, int split, int P, int* __restrict__ twin,
                              double* __restrict__ loss) {
  __shared__ double best[kThreads];
  double tot = 0.0;
  for (int b0 = 0; b0 < count; b0 += kThreads) {
    const int b = b0 + threadIdx.x;
    if (b < count) {
      double a = 0.0, t = 0.0;
#pragma unroll 8
      for (int z = 0; z < split; ++z) {
        const double2 v = reinterpret_cast<const double2*>(part)[(long long)b * split + z];
        a += v.x;
        t += v.y;
      }
      twin[b] = t < a ? 1 : 0;
      best[threadIdx.x] = (t < a ? t : a) / P;
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int k = 0; k < min(kThreads, count - b0); ++k) tot += best[k];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = tot / count;
}

// dL/d(head output) for the chosen branch -> BF16 [M][8] (channels 4..7 zero),
// and the head bias gradient's partial sums over the CTA's pixels
__global__ void __launch_bounds__(kThreads) k_loss_grad(const float* __restrict__ out, const float* __restrict__ amp_t,
                                                        const float* __restrict__ ph_t, const float* __restrict__ sup_t,
                                                        const int* __restrict__ twin, int n, int count, float ws,
                                                        __nv_bfloat16* __restrict__ dout_b, double* __restrict__ bpart) {
  const int P = n * n;
  const long long total = (long long)count * P;
  const float sc = 1.f / ((float)P * count);
  double sum[4] = {0.0, 0.0, 0.0, 0.0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int b = (int)(i / P), p = (int)(i - (long long)b * P);
    int q = p;
    float sg = 1.f;
    if (twin[b]) {
      const int y = p / n, x = p - y * n;
      q = ((n - y) % n) * n + (n - x) % n;
      sg = -1.f;
    }
    const long long t = (long long)b * P + q;
    const float at = amp_t[t], pt = sg * ph_t[t], st = sup_t[t];
    float s, c;
    sincosf(pt, &s, &c);
    const float4 o = *reinterpret_cast<const float4*>(out + i * 8);
    float g[8] = {};
    g[0] = 2.f * (o.x - at) * sc;
    g[1] = 2.f * at * (o.y - c) * sc;
    g[2] = 2.f * at * (o.z - s) * sc;
    g[3] = ws * (sigmoidf_(o.w) - st) * sc;
#pragma unroll
    for (int k = 0; k < 4; ++k) sum[k] += g[k];
    st8(dout_b + i * 8, g);
  }
  __shared__ double r[kThreads / 32][4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_down_sync(0xffffffffu, sum[k], o);
    if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5][k] = sum[k];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double s = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) s += r[w][threadIdx.x];
    bpart[blockIdx.x * 4 + threadIdx.x] = s;
  }
}

// head bias gradient: one warp per channel over the CTAs' partial sums (fixed order)
__global__ void k_bias_grad(const double* __restrict__ bpart, int nblk, float* __restrict__ gb) {
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double s = 0.0;
  for (int i = lane; i < nblk; i += 32) s += bpart[i * 4 + c];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) gb[c] = (float)s;
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       long long count, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count; i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// network output [b][p][8] -> user [b][4][n][n]
__global__ void k_head_out(const float* __restrict__ o, int P, long long total, float* __restrict__ out) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long b = i / P;
    const int p = (int)(i - b * P);
#pragma unroll
    for (int c = 0; c < 4; ++c) out[(b * 4 + c) * P + p] = o[i * 8 + c];
  }
}
// user layout [b][4][n][n] -> [b][p][8]
__global__ void k_head_in(const float* __restrict__ in, int P, long long total, float* __restrict__ o) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long b = i / P;
    const int p = (int)(i - b * P);
#pragma unroll
    for (int c = 0; c < 4; ++c) o[i * 8 + c] = in[(b * 4 + c) * P + p];
  }
}

// rho0 (complex, the object frame: the object centred in the array as the
// reference keeps objectWave) and the support from the network output: the
// predicted mask (logit > 0) dilated by `dil` pixels (a square window), since
// HIO tolerates a loose support but not one that cuts into the object
__global__ void k_warm_object(const float* __restrict__ out, int n, int dil, long long total, float2* __restrict__ rho,
                              float* __restrict__ sup) {
  const int P = n * n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long b = i / P;
    const int q = (int)(i - b * P);
    const int y = q / n, x = q - y * n;
    const float* o = out + b * 4 * P;
    const float a = fmaxf(o[q], 0.f), c = o[P + q], s = o[2 * P + q], lg = o[3 * P + q];
    bool in = false;
    for (int dy = -dil; dy <= dil && !in; ++dy) {
      const int yy = y + dy;
      if (yy < 0 || yy >= n) continue;
      for (int dx = -dil; dx <= dil; ++dx) {
        const int xx = x + dx;
        if (xx >= 0 && xx < n && o[3 * P + yy * n + xx] > 0.f) {
          in = true;
          break;
        }
      }
    }
    const float r = hypotf(c, s);
    float2 v = make_float2(0.f, 0.f);
    if (lg > 0.f) v = r > 0.f ? make_float2(a * c / r, a * s / r) : make_float2(a, 0.f);
    rho[i] = v;
    sup[i] = in ? 1.f : 0.f;
  }
}

// psi0 = sqrt(I) e^{i arg F}
__global__ void k_warm_psi(const float2* __restrict__ F, const float* __restrict__ inten, long long total,
                           float2* __restrict__ psi) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const float a = sqrtf(fmaxf(inten[i], 0.f));
    const float2 f = F[i];
    const float r = hypotf(f.x, f.y);
    psi[i] = r > 0.f ? make_float2(a * f.x / r, a * f.y / r) : make_float2(a, 0.f);
  }
}

// --------------------------------------------------------------------- host
inline int grid_for(long long total, int threads = kThreads) {
  long long b = (total + threads - 1) / threads;
  const long long cap = sm_count() * 16LL;
  return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

enum { L_CONV = 0, L_CONVT = 1, L_HEAD = 2 };

struct Layer {
  int kind;
  int cin_r, cin_p, cout_r, cout_p;   // layer channels (real / padded)
  int c0;                             // channels of input part 0 (concat)
  int k, s, p;                        // kernel, stride, padding
  int in_h, out_h;                    // spatial sizes
  long long w_off = -1, g_off = -1, b_off = -1, bias_off = -1;
  // underlying convolution weight: [co][k][k][ci] with (co, ci) = (cout, cin) for a
  // convolution and (cin, cout) for a transposed one
  int wco_r, wci_r, wco_p, wci_p;
  __nv_bfloat16 *wb = nullptr, *wt = nullptr;
  __nv_bfloat16 *pb = nullptr, *pt = nullptr;   // the same, packed for k_conv_umma
  int in0 = -1, in1 = -1;             // producer layers (-1: the network input)
  float* pre = nullptr;               // conv output (FP32)
  __nv_bfloat16* act = nullptr;       // activation (BF16)
  float* stats = nullptr;             // mean, rstd per (pattern, group)
  float* dact = nullptr;              // gradient of the activation (FP32)
  __nv_bfloat16* dpre = nullptr;      // gradient of the conv output (BF16)
};

struct Net {
  cdx_unet_config cfg;
  cudaStream_t st = nullptr;
  bool own_stream = false;
  std::vector<Layer> L;
  long long np = 0;
  float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
  __nv_bfloat16* x_in = nullptr;
  std::vector<void*> allocs;
  float* wpart = nullptr;
  size_t wpart_cap = 0;
  double *gpart = nullptr, *cpart = nullptr, *lpart = nullptr, *loss = nullptr;
  size_t gpart_cap = 0, cpart_cap = 0;
  double* bpart = nullptr; // head bias gradient partials
  unsigned* mx = nullptr;  // largest log(1 + I) per pattern, float bits
  int* twin = nullptr;
  float2* wrk = nullptr;   // warm start scratch
  int* umma_err = nullptr; // set by a tcgen05 tile whose pipeline wait timed out (check_umma)
  int adam_t = 0;
  bool dep = false;        // launch the forward's kernels dependently (small passes)
  bool weights_dirty = true;
};

template <typename T>
int dalloc(Net* u, T** p, size_t count) {
  void* q = nullptr;
  cudaError_t e = cudaMalloc(&q, count * sizeof(T) + 16);
  if (e != cudaSuccess) return set_error(CDX_ERR_NOMEM, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  u->allocs.push_back(q);
  *p = (T*)q;
  return CDX_OK;
}

const __nv_bfloat16* act_of(const Net* u, int idx) { return idx < 0 ? u->x_in : u->L[idx].act; }
int chan_of(const Net* u, int idx) { return idx < 0 ? 8 : u->L[idx].cout_p; }

int build(Net* u) {
  const cdx_unet_config& c = u->cfg;
  const int B = c.batch;
  auto add = [&](int kind, int in0, int in1, int cin_r, int cout_r, int k, int s, int p, int in_h) {
    Layer l{};
    l.kind = kind;
    l.in0 = in0;
    l.in1 = in1;
    l.cin_r = cin_r;
    l.cin_p = in0 < 0 ? 8 : cin_r;
    l.c0 = in1 >= 0 ? chan_of(u, in0) : l.cin_p;
    l.cout_r = cout_r;
    l.cout_p = kind == L_HEAD ? 8 : cout_r;
    l.k = k;
    l.s = s;
    l.p = p;
    l.in_h = in_h;
    l.out_h = kind == L_CONVT ? in_h * 2 : (in_h + 2 * p - k) / s + 1;
    if (kind == L_CONVT) {
      l.wco_r = cin_r; l.wci_r = cout_r; l.wco_p = cin_r; l.wci_p = cout_r;
    } else {
      l.wco_r = cout_r; l.wci_r = in0 < 0 ? 1 : cin_r; l.wco_p = l.cout_p; l.wci_p = l.cin_p;
    }
    l.w_off = u->np;
    u->np += (long long)l.wco_r * k * k * l.wci_r;
    if (kind != L_HEAD) {
      l.g_off = u->np; u->np += cout_r;
      l.b_off = u->np; u->np += cout_r;
    } else {
      l.bias_off = u->np; u->np += 4;
    }
    u->L.push_back(l);
    return (int)u->L.size() - 1;
  };
  std::vector<int> skip(c.levels);
  int h = c.n, ch = c.base;
  int cur = add(L_CONV, -1, -1, 1, ch, 3, 1, 1, h);
  cur = add(L_CONV, cur, -1, ch, ch, 3, 1, 1, h);
  skip[0] = cur;
  for (int l = 1; l < c.levels; ++l) {
    cur = add(L_CONV, cur, -1, ch, ch * 2, 3, 2, 1, h);
    h /= 2;
    ch *= 2;
    cur = add(L_CONV, cur, -1, ch, ch, 3, 1, 1, h);
    skip[l] = cur;
  }
  for (int l = c.levels - 2; l >= 0; --l) {
    const int up = add(L_CONVT, cur, -1, ch, ch / 2, 2, 2, 0, h);
    h *= 2;
    ch /= 2;
    cur = add(L_CONV, up, skip[l], 2 * ch, ch, 3, 1, 1, h);
  }
  add(L_HEAD, cur, -1, ch, 4, 1, 1, 0, h);
  // buffers
  int e;
  if ((e = dalloc(u, &u->params, u->np)) || (e = dalloc(u, &u->grads, u->np)) || (e = dalloc(u, &u->m, u->np)) ||
      (e = dalloc(u, &u->v, u->np)))
    return e;
  if ((e = dalloc(u, &u->x_in, (size_t)B * c.n * c.n * 8))) return e;
  size_t gp = 0, cp = 0, wp = 0;
  for (auto& l : u->L) {
    const size_t px = (size_t)B * l.out_h * l.out_h;
    const size_t wsz = (size_t)l.wco_p * l.k * l.k * l.wci_p;
    if ((e = dalloc(u, &l.wb, wsz)) || (e = dalloc(u, &l.wt, wsz)) || (e = dalloc(u, &l.pb, wsz)) ||
        (e = dalloc(u, &l.pt, wsz)))
      return e;
    if ((e = dalloc(u, &l.pre, px * l.cout_p)) || (e = dalloc(u, &l.act, px * l.cout_p)) ||
        (e = dalloc(u, &l.dact, px * l.cout_p)) || (e = dalloc(u, &l.dpre, px * l.cout_p)))
      return e;
    if (l.kind != L_HEAD && (e = dalloc(u, &l.stats, (size_t)B * c.groups * 2))) return e;
    gp = std::max(gp, (size_t)B * c.groups * 64 * 2);
    cp = std::max(cp, (size_t)B * 64 * l.cout_p * 2);
    wp = std::max(wp, (size_t)64 * wsz);
  }
  if ((e = dalloc(u, &u->gpart, gp)) || (e = dalloc(u, &u->cpart, cp)) || (e = dalloc(u, &u->wpart, wp)) ||
      (e = dalloc(u, &u->mx, (size_t)B)) || (e = dalloc(u, &u->lpart, (size_t)B * 64 * 2)) ||
      (e = dalloc(u, &u->loss, 1)) || (e = dalloc(u, &u->bpart, (size_t)4 * 16 * sm_count())) ||
      (e = dalloc(u, &u->twin, (size_t)B)) || (e = dalloc(u, &u->wrk, (size_t)B * c.n * c.n)) ||
      (e = dalloc(u, &u->umma_err, 1)))
    return e;
  u->gpart_cap = gp;
  u->cpart_cap = cp;
  u->wpart_cap = wp;
  return CDX_OK;
}

// He-normal weights from a SplitMix64 stream, GroupNorm gamma 1 / beta 0, head bias 0
void init_params(Net* u, std::vector<float>& h) {
  h.assign(u->np, 0.f);
  uint64_t s = u->cfg.seed * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
  auto next = [&]() {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  auto unif = [&]() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); };
  for (auto& l : u->L) {
    const long long cnt = (long long)l.wco_r * l.k * l.k * l.wci_r;
    const double fan_in = l.kind == L_CONVT ? (double)l.cin_r : (double)l.k * l.k * l.wci_r;
    const double sd = l.kind == L_HEAD ? std::sqrt(1.0 / fan_in) : std::sqrt(2.0 / fan_in);
    for (long long i = 0; i < cnt; ++i) {
      const double r = std::sqrt(-2.0 * std::log(unif())), t = 6.283185307179586 * unif();
      h[l.w_off + i] = (float)(sd * r * std::cos(t));
    }
    if (l.g_off >= 0)
      for (int i = 0; i < l.cout_r; ++i) h[l.g_off + i] = 1.f;
  }
}

int refresh_weights(Net* u) {
  if (!u->weights_dirty) return CDX_OK;
  for (auto& l : u->L) {
    const long long tot = (long long)l.wco_p * l.k * l.k * l.wci_p;
    k_weights_bf16<<<grid_for(tot), kThreads, 0, u->st>>>(u->params + l.w_off, l.wco_r, l.wci_r, l.wco_p, l.wci_p,
                                                           l.k * l.k, l.wb, l.wt, l.pb, l.pt);
  }
  U_CK(cudaGetLastError());
  u->weights_dirty = false;
  return CDX_OK;
}

// the underlying convolution of a layer (for a transposed layer: from its output to its input)
ConvShape conv_shape(const Net* u, const Layer& l, int count) {
  ConvShape s{};
  s.N = count;
  s.KH = s.KW = l.k;
  s.S = l.s;
  s.P = l.p;
  if (l.kind == L_CONVT) {
    s.H = s.W = l.out_h;
    s.Cin = s.C0 = l.cout_p;
    s.Ho = s.Wo = l.in_h;
    s.Cout = l.cin_p;
  } else {
    s.H = s.W = l.in_h;
    s.Cin = l.cin_p;
    s.C0 = l.c0;
    s.Ho = s.Wo = l.out_h;
    s.Cout = l.cout_p;
  }
  (void)u;
  return s;
}

template <int BN, class Op>
int launch_umma(const Op& op, long long M, int NC, int K, int* err, cudaStream_t st) {
  const cudaError_t e = umma::launch_ps<BN, Op>(op, (int)M, NC, K, err, st);
  U_CK(e);
  return CDX_OK;
}

// The convolution (or its data gradient) on k_conv_umma, where the layer fits it:
// 3x3 and 2x2 layers of 16 to 256 channels in and out.
template <bool DGRAD>
bool plan_umma(const GemmArgs& g, const __nv_bfloat16* packed, ConvUmma& a, int& smem) {
  const ConvShape& s = g.s;
  a = ConvUmma{};
  a.w = packed;
  a.nimg = s.N;
  a.acc0 = g.acc0;
  a.acc1 = g.acc1;
  a.out0 = g.out0;
  const bool k3 = s.KH == 3 && s.KW == 3 && s.P == 1, k2 = s.KH == 2 && s.KW == 2 && s.P == 0;
  if (!DGRAD) {
    a.x0 = g.x0; a.x1 = g.x1; a.C0 = s.C0; a.C = s.Cin;
    a.N = a.N0 = s.Cout;
    a.out1 = g.out0;
    a.H = s.H; a.W = s.W; a.GH = a.OH = s.Ho; a.GW = a.OW = s.Wo;
    if (k3 && s.S == 1) cu_conv3(a, false);
    else if (k3 && s.S == 2) cu_conv_s2(a, 3, 1);
    else if (k2 && s.S == 2) cu_conv_s2(a, 2, 0);
    else return false;
  } else {
    a.x0 = a.x1 = g.dy; a.C0 = a.C = s.Cout;
    a.N = s.Cin; a.N0 = s.C0;
    a.out1 = g.out1;
    a.H = a.GH = s.Ho; a.W = a.GW = s.Wo; a.OH = s.H; a.OW = s.W;
    if (k3 && s.S == 1) cu_conv3(a, true);
    else if (s.S == 2 && s.H == 2 * s.Ho && s.W == 2 * s.Wo && (k3 || k2)) cu_adj_s2(a, s.KH, s.P);
    else return false;
  }
  return cu_plan(a, s.KH * s.KW, smem);
}

// cdx_unet_config::umma 2 and 3: every convolution and weight gradient on the gathering kernels
bool gather_all(const Net* u) { return u->cfg.umma == 2 || u->cfg.umma == 3; }

// forward (DGRAD false) or data-gradient GEMM: k_conv_umma where the layer fits it (`packed`:
// its weights); else the gathering kernels, tcgen05 when the net is configured for them
template <bool DGRAD>
int launch_gemm(const Net* u, const GemmArgs& a, const __nv_bfloat16* packed, cudaStream_t st) {
  const ConvShape& s = a.s;
  ConvUmma c;
  int smem = 0;
  if (!gather_all(u) && plan_umma<DGRAD>(a, packed, c, smem)) {
    U_CK(launch_conv_umma(c, smem, u->umma_err, u->dep, st));
    return CDX_OK;
  }
  const long long M = DGRAD ? (long long)s.N * s.H * s.W : (long long)s.N * s.Ho * s.Wo;
  const int NC = DGRAD ? s.Cin : s.Cout;
  const int K = DGRAD ? s.KH * s.KW * s.Cout : s.KH * s.KW * s.Cin;
  if (u->cfg.umma != 0 && u->cfg.umma != 2) {
    using Op = typename std::conditional<DGRAD, ConvDgradOp, ConvFwdOp>::type;
    const Op op{a};
    if (NC <= 32) return launch_umma<32>(op, M, NC, K, u->umma_err, st);
    if (NC <= 64) return launch_umma<64>(op, M, NC, K, u->umma_err, st);
    return launch_umma<128>(op, M, NC, K, u->umma_err, st);
  }
  const dim3 grid((unsigned)((M + 127) / 128), (unsigned)((NC + (NC <= 32 ? 31 : 63)) / (NC <= 32 ? 32 : 64)));
  U_CK(net_launch(u->dep, NC <= 32 ? k_conv_gemm<DGRAD, 32> : k_conv_gemm<DGRAD, 64>, grid, 128, 0, st, a));
  return CDX_OK;
}

int launch_wgrad(Net* u, GemmArgs a, const Layer& l) {
  const ConvShape& s = a.s;
  const long long M = (long long)s.N * s.Ho * s.Wo;
  const int K = s.KH * s.KW * s.Cin;
  const int tx = (K + 63) / 64, ty = (s.Cout + 63) / 64;
  long long splits = (sm_count() * 4LL + tx * ty - 1) / (tx * ty);
  splits = std::max(1LL, std::min(splits, std::min(64LL, (M + 255) / 256)));
  long long mps = (M + splits - 1) / splits;
  mps = (mps + 31) / 32 * 32;
  splits = (M + mps - 1) / mps;
  if ((size_t)(splits * s.Cout * K) > u->wpart_cap) return set_error(CDX_ERR_STATE, "wgrad scratch too small");
  a.out0 = u->wpart;
  a.m_per_split = (int)mps;
  WgradUmma w{};
  w.x0 = a.x0; w.x1 = a.x1; w.dy = a.dy; w.part = u->wpart;
  w.C0 = s.C0; w.Cin = s.Cin; w.Cout = s.Cout;
  w.H = s.H; w.W = s.W; w.Ho = s.Ho; w.Wo = s.Wo;
  w.KH = s.KH; w.KW = s.KW; w.S = s.S; w.P = s.P;
  w.M = (int)M;
  w.m_per_split = (int)mps;
  if (!gather_all(u) && wg_plan(w, (int)splits, sm_count())) U_CK(launch_wgrad_umma(w, (int)splits, u->umma_err, u->st));
  else k_conv_wgrad<<<dim3(tx, ty, (unsigned)splits), 128, 0, u->st>>>(a);
  const long long tot = (long long)l.wco_r * l.k * l.k * l.wci_r;
  k_wgrad_reduce<<<grid_for(tot), kThreads, 0, u->st>>>(u->wpart, (int)splits, l.wco_r, l.wci_r, l.wco_p, l.wci_p,
                                                         l.k * l.k, u->grads + l.w_off);
  U_CK(cudaGetLastError());
  return CDX_OK;
}

int gn_split(const Net* u, int HW, int count) {
  const int ng = count * u->cfg.groups;
  int sp = (sm_count() * 4 + ng - 1) / ng;
  sp = std::max(1, std::min(sp, std::min(64, HW / 64 > 0 ? HW / 64 : 1)));
  return sp;
}

// grid of the element-wise GroupNorm kernels: about eight CTAs per SM, at least four pixels a thread
dim3 gn_grid(int HW, int C, int count) {
  const int oc = gn_octs(C), per = kThreads / oc * 4;
  const int x = std::max(1, std::min((HW + per - 1) / per, sm_count() * 8 / count));
  return dim3(count, x, (C / 8 + oc - 1) / oc);
}

int forward(Net* u, const float* inten, int count) {
  const cdx_unet_config& c = u->cfg;
  int e = refresh_weights(u);
  if (e) return e;
  u->dep = (long long)count * c.n * c.n <= 1LL << 20;
  U_CK(cudaMemsetAsync(u->mx, 0, sizeof(unsigned) * count, u->st));
  const int P = c.n * c.n;
  const dim3 pgrid(count, std::max(1, std::min((P + kThreads - 1) / kThreads, sm_count() * 8 / count)));
  k_prep_max<<<pgrid, kThreads, 0, u->st>>>(inten, P, u->mx);
  U_CK(net_launch(u->dep, k_prep_input, pgrid, kThreads, 0, u->st, inten, u->mx, u->x_in, c.n));
  for (auto& l : u->L) {
    GemmArgs a{};
    a.s = conv_shape(u, l, count);
    if (l.kind == L_CONVT) {
      a.dy = act_of(u, l.in0);
      a.w = l.wt;
      a.out0 = l.pre;
      a.out1 = l.pre;
      if ((e = launch_gemm<true>(u, a, l.pt, u->st))) return e;
    } else {
      a.x0 = act_of(u, l.in0);
      a.x1 = l.in1 >= 0 ? act_of(u, l.in1) : a.x0;
      a.w = l.wb;
      a.out0 = l.pre;
      if ((e = launch_gemm<false>(u, a, l.pb, u->st))) return e;
    }
    const long long px = (long long)count * l.out_h * l.out_h;
    if (l.kind == L_HEAD) {
      k_bias_add<<<grid_for(px * 4), kThreads, 0, u->st>>>(l.pre, u->params + l.bias_off, px);
      continue;
    }
    const int HW = l.out_h * l.out_h, sp = gn_split(u, HW, count), C = l.cout_p, gpc = gn_groups(C / c.groups, c.groups);
    U_CK(net_launch(u->dep, k_gn_stats, dim3(count, sp, c.groups / gpc), kThreads / 4 * gpc, gpc * kThreads * sizeof(double),
                    u->st, l.pre, HW, C, c.groups, gpc, sp, u->gpart));
    U_CK(net_launch(u->dep, k_gn_apply, gn_grid(HW, C, count), kThreads, c.groups * sizeof(float2), u->st, l.pre, u->gpart, sp,
                    l.stats, u->params + l.g_off, u->params + l.b_off, HW, C, c.groups, c.slope, l.act));
  }
  U_CK(cudaGetLastError());
  return CDX_OK;
}

int backward(Net* u, const float* amp_t, const float* ph_t, const float* sup_t, int count) {
  const cdx_unet_config& c = u->cfg;
  const Layer& head = u->L.back();
  const int P = c.n * c.n;
  u->dep = false;
  // the first data gradient that reaches a layer's activation is stored, later ones are added
  std::vector<char> reached(u->L.size(), 0);
  const int lsp = std::max(1, std::min(64, (sm_count() * 4 + count - 1) / count));
  k_loss_partial<<<dim3(count, lsp), kThreads, 0, u->st>>>(head.pre, amp_t, ph_t, sup_t, c.n, lsp, c.support_weight,
                                                            u->lpart);
  k_loss_select<<<1, kThreads, 0, u->st>>>(u->lpart, count, lsp, P, u->twin, u->loss);
  const int gl = grid_for((long long)count * P);
  k_loss_grad<<<gl, kThreads, 0, u->st>>>(head.pre, amp_t, ph_t, sup_t, u->twin, c.n, count, c.support_weight,
                                          head.dpre, u->bpart);
  k_bias_grad<<<1, 128, 0, u->st>>>(u->bpart, gl, u->grads + head.bias_off);
  int e;
  for (int li = (int)u->L.size() - 1; li >= 0; --li) {
    Layer& l = u->L[li];
    const int HW = l.out_h * l.out_h;
    if (l.kind != L_HEAD) {
      const int sp = gn_split(u, HW, count);
      if ((size_t)count * sp * l.cout_p * 2 > u->cpart_cap) return set_error(CDX_ERR_STATE, "GroupNorm scratch too small");
      const int C = l.cout_p, gpc = gn_groups(C / c.groups, c.groups);
      k_gn_bwd_stats<<<dim3(count, sp, c.groups / gpc), kThreads / 4 * gpc, gpc * kThreads * sizeof(double), u->st>>>(
          l.pre, l.dact, l.stats, u->params + l.g_off, u->params + l.b_off, HW, C, c.groups, gpc, sp, c.slope, u->gpart,
          u->cpart);
      k_gn_bwd_finalize<<<(C + 7) / 8, 256, 0, u->st>>>(u->cpart, count * sp, C, u->grads + l.g_off,
                                                        u->grads + l.b_off);
      k_gn_bwd_apply<<<gn_grid(HW, C, count), kThreads, c.groups * sizeof(float4), u->st>>>(
          l.pre, l.dact, l.stats, u->gpart, sp, u->params + l.g_off, u->params + l.b_off, HW, C, c.groups, c.slope,
          l.dpre);
    }
    GemmArgs a{};
    a.s = conv_shape(u, l, count);
    if (l.kind == L_CONVT) {
      // weight gradient: wgrad of the underlying convolution with X = dz, dY = this layer's input
      a.x0 = l.dpre;
      a.x1 = l.dpre;
      a.dy = act_of(u, l.in0);
      if ((e = launch_wgrad(u, a, l))) return e;
      if (l.in0 >= 0) {
        GemmArgs f{};
        f.s = a.s;
        f.x0 = l.dpre;
        f.x1 = l.dpre;
        f.w = l.wb;
        f.out0 = u->L[l.in0].dact;
        f.acc0 = reached[l.in0];
        reached[l.in0] = 1;
        if ((e = launch_gemm<false>(u, f, l.pb, u->st))) return e;
      }
    } else {
      a.x0 = act_of(u, l.in0);
      a.x1 = l.in1 >= 0 ? act_of(u, l.in1) : a.x0;
      a.dy = l.dpre;
      if ((e = launch_wgrad(u, a, l))) return e;
      if (l.in0 >= 0) {
        GemmArgs d{};
        d.s = a.s;
        d.dy = l.dpre;
        d.w = l.wt;
        d.out0 = u->L[l.in0].dact;
        d.out1 = l.in1 >= 0 ? u->L[l.in1].dact : d.out0;
        d.acc0 = reached[l.in0];
        reached[l.in0] = 1;
        if (l.in1 >= 0) {
          d.acc1 = reached[l.in1];
          reached[l.in1] = 1;
        }
        if ((e = launch_gemm<true>(u, d, l.pt, u->st))) return e;
      }
    }
  }
  U_CK(cudaGetLastError());
  return CDX_OK;
}

}  // namespace unet
}  // namespace cdx

using namespace cdx;
using namespace cdx::unet;

struct cdx_unet {
  Net net;
};

extern "C" {

int cdx_unet_config_default(cdx_unet_config* c) {
  if (!c) return set_error(CDX_ERR_ARG, "null config");
  c->n = 256;
  c->levels = 4;
  c->base = 32;
  c->batch = 64;
  c->groups = 8;
  c->slope = 0.01f;
  c->support_weight = 0.1f;
  c->seed = 20260101ull;
  c->umma = 0;
  return CDX_OK;
}

int cdx_unet_create(const cdx_unet_config* c, void* stream, cdx_unet** out) {
  if (!c || !out) return set_error(CDX_ERR_ARG, "null argument");
  *out = nullptr;
  if (c->levels < 2 || c->levels > 8) return set_error(CDX_ERR_ARG, "levels must be in [2, 8]");
  if (c->base < 8 || c->base % 8) return set_error(CDX_ERR_ARG, "base must be a positive multiple of 8");
  if (c->groups < 1 || c->base % c->groups || (kThreads % (c->base / c->groups)) ||
      c->base / c->groups > kThreads)
    return set_error(CDX_ERR_ARG, "groups must divide base (and base/groups divide 256)");
  // the statistics kernels give each of a group's channels a thread of 256 (channels double per level)
  if (((long long)(c->base / c->groups) << (c->levels - 1)) > kThreads)
    return set_error(CDX_ERR_ARG, "a group may hold at most 256 channels at the deepest level "
                                  "(base/groups * 2^(levels-1))");
  if (c->n < 16 || c->n % (8 << (c->levels - 1))) return set_error(CDX_ERR_SIZE, "n must be a multiple of 8*2^(levels-1)");
  if (c->batch < 1) return set_error(CDX_ERR_ARG, "batch must be >= 1");
  if (!cdx_size_supported(c->n)) return set_error(CDX_ERR_SIZE, "n is not a supported FFT length");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    return set_error(CDX_ERR_NOLIB, "no CUDA device");
  }
  cdx_unet* u = new cdx_unet();
  Net* n = &u->net;
  n->cfg = *c;
  if (stream) {
    n->st = (cudaStream_t)stream;
  } else {
    if (cudaStreamCreateWithFlags(&n->st, cudaStreamNonBlocking) != cudaSuccess) {
      delete u;
      return set_error(CDX_ERR_CUDA, "stream create failed");
    }
    n->own_stream = true;
  }
  int e = build(n);
  // the element-wise GroupNorm kernels hold a pattern's group statistics (16 bytes a group at most)
  for (const void* k : {(const void*)k_gn_apply, (const void*)k_gn_bwd_apply})
    if (!e && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024) != cudaSuccess)
      e = set_error(CDX_ERR_CUDA, "kernel attributes");
  if (!e) {
    std::vector<float> h;
    init_params(n, h);
    if (cudaMemcpy(n->params, h.data(), sizeof(float) * h.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(n->m, 0, sizeof(float) * n->np) != cudaSuccess ||
        cudaMemset(n->v, 0, sizeof(float) * n->np) != cudaSuccess ||
        cudaMemset(n->grads, 0, sizeof(float) * n->np) != cudaSuccess ||
        cudaMemset(n->umma_err, 0, sizeof(int)) != cudaSuccess)
      e = set_error(CDX_ERR_CUDA, "parameter upload failed");
  }
  if (e) {
    cdx_unet_destroy(u);
    return e;
  }
  *out = u;
  return CDX_OK;
}

void cdx_unet_destroy(cdx_unet* u) {
  if (!u) return;
  Net* n = &u->net;
  if (n->st) cudaStreamSynchronize(n->st);
  for (void* p : n->allocs) cudaFree(p);
  if (n->own_stream && n->st) cudaStreamDestroy(n->st);
  delete u;
}

long long cdx_unet_param_count(const cdx_unet* u) { return u ? u->net.np : -1; }

int cdx_unet_get_params(const cdx_unet* u, float* host, long long count) {
  if (!u || !host || count != u->net.np) return set_error(CDX_ERR_ARG, "bad parameter buffer");
  U_CK(cudaStreamSynchronize(u->net.st));
  U_CK(cudaMemcpy(host, u->net.params, sizeof(float) * count, cudaMemcpyDeviceToHost));
  return CDX_OK;
}

int cdx_unet_set_params(cdx_unet* u, const float* host, long long count) {
  if (!u || !host || count != u->net.np) return set_error(CDX_ERR_ARG, "bad parameter buffer");
  U_CK(cudaStreamSynchronize(u->net.st));
  U_CK(cudaMemcpy(u->net.params, host, sizeof(float) * count, cudaMemcpyHostToDevice));
  u->net.weights_dirty = true;
  return CDX_OK;
}

int cdx_unet_get_grads(const cdx_unet* u, float* host, long long count) {
  if (!u || !host || count != u->net.np) return set_error(CDX_ERR_ARG, "bad gradient buffer");
  U_CK(cudaStreamSynchronize(u->net.st));
  U_CK(cudaMemcpy(host, u->net.grads, sizeof(float) * count, cudaMemcpyDeviceToHost));
  return CDX_OK;
}

// A wait that ran out in this call's kernels is reported here and cleared for the next call's.
static int check_umma(Net* n) {
  int flag = 0;
  U_CK(cudaMemcpyAsync(&flag, n->umma_err, sizeof(int), cudaMemcpyDeviceToHost, n->st));
  U_CK(cudaStreamSynchronize(n->st));
  if (flag) {
    U_CK(cudaMemsetAsync(n->umma_err, 0, sizeof(int), n->st));
    return set_error(CDX_ERR_CUDA, "tensor-core GEMM pipeline wait timed out");
  }
  return CDX_OK;
}

int cdx_unet_forward(cdx_unet* u, const float* intensity, float* out, int count) {
  if (!u || !intensity || !out) return set_error(CDX_ERR_ARG, "null argument");
  if (count < 1 || count > u->net.cfg.batch) return set_error(CDX_ERR_ARG, "count must be in [1, batch]");
  Net* n = &u->net;
  int e = forward(n, intensity, count);
  if (e) return e;
  const int P = n->cfg.n * n->cfg.n;
  k_head_out<<<grid_for((long long)count * P), kThreads, 0, n->st>>>(n->L.back().pre, P, (long long)count * P, out);
  U_CK(cudaGetLastError());
  return check_umma(n);
}

int cdx_unet_loss_backward(cdx_unet* u, const float* intensity, const float* amp_t, const float* phase_t,
                           const float* support_t, int count, double* loss) {
  if (!u || !intensity || !amp_t || !phase_t || !support_t) return set_error(CDX_ERR_ARG, "null argument");
  if (count < 1 || count > u->net.cfg.batch) return set_error(CDX_ERR_ARG, "count must be in [1, batch]");
  Net* n = &u->net;
  int e = forward(n, intensity, count);
  if (e) return e;
  if ((e = backward(n, amp_t, phase_t, support_t, count))) return e;
  if (loss) {
    U_CK(cudaMemcpyAsync(loss, n->loss, sizeof(double), cudaMemcpyDeviceToHost, n->st));
  }
  return check_umma(n);
}

int cdx_unet_adam_step(cdx_unet* u, float lr) {
  if (!u) return set_error(CDX_ERR_ARG, "null network");
  Net* n = &u->net;
  n->adam_t += 1;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.f - (float)std::pow((double)b1, n->adam_t), c2 = 1.f - (float)std::pow((double)b2, n->adam_t);
  k_adam<<<grid_for(n->np), kThreads, 0, n->st>>>(n->params, n->grads, n->m, n->v, n->np, lr, b1, b2, 1e-8f, c1, c2);
  U_CK(cudaGetLastError());
  n->weights_dirty = true;
  return CDX_OK;
}

int cdx_unet_warm_start(cdx_unet* u, const float* intensity, const float* out, int count, int dilate, void* psi0,
                        float* support) {
  if (!u || !intensity || !out || !psi0 || !support) return set_error(CDX_ERR_ARG, "null argument");
  if (dilate < 0 || dilate > 16) return set_error(CDX_ERR_ARG, "dilate must be in [0, 16]");
  Net* n = &u->net;
  if (count < 1 || count > n->cfg.batch) return set_error(CDX_ERR_ARG, "count must be in [1, batch]");
  const int N = n->cfg.n;
  const long long tot = (long long)count * N * N;
  k_warm_object<<<grid_for(tot), kThreads, 0, n->st>>>(out, N, dilate, tot, n->wrk, support);
  U_CK(cudaGetLastError());
  int e = cdx_fft2(n->wrk, n->wrk, N, N, count, 0, n->st);
  if (e) return e;
  k_warm_psi<<<grid_for(tot), kThreads, 0, n->st>>>(n->wrk, intensity, tot, (float2*)psi0);
  U_CK(cudaGetLastError());
  U_CK(cudaStreamSynchronize(n->st));
  return CDX_OK;
}

}  // extern "C"
