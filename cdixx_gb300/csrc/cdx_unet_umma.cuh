// The U-Net's forward and data-gradient convolutions as tcgen05 GEMMs on halo
// patches (sm_103a).
//
// A CTA computes 128 pixels (16 rows x 8 columns of a tile grid) x all N output
// channels.  The input pixels its taps touch are staged once, as planes of eight
// channels: plane c8, slot s holds the 16 bytes of one patch pixel.  Eight
// consecutive slots are then one core matrix of the K-major no-swizzle operand
// layout, rows of the tile grid are the 8-row groups (stride SBO), and a tap is
// nothing but another start address, so the nine taps of a 3x3 read the same patch
// (im2col gathers, one copy of every tap, kept the copy path busier than the tensor
// core: cdx_unet_gemm.cuh).  Stride-2 convolutions split the patch columns by parity
// so that the pixels of a tap are consecutive slots; their data gradients and the
// transposed convolutions run one GEMM per output parity class on the taps that
// reach it, four on one patch.  The weights come packed as [K/8][N][8], a stage is
// one bulk copy; layers whose packed weights fit stay resident for all tiles of the
// (persistent) CTA.
//
// K runs over taps in order, then channels, in steps of 16, as in k_conv_gemm: the
// sums are the same, bit for bit.
//
// Roles (320 threads): warps 0-3 copy patches (cp.async), 4-7 drain the accumulators
// (two, in TMEM), warp 8 issues the MMAs, warp 9 the weight copies.  Every wait is
// bounded; a role that gives up sets *err and the abort flag, which ends the others.
//
// Bound by HBM and the L2 (FP32 outputs, patches and streamed weights), and before that by
// the MMA lane: one thread issues every MMA, and a loop that builds both descriptors
// each time spent 130-190 cycles per MMA on it.  The loops below add to descriptors
// built once and are unrolled: batch 32 of 256^2 (4 levels, 32 channels), the step's 26
// launches 3.02 -> 2.60 ms (10.5 with the gathering kernels), 32 -> 32 channels at 256^2
// 113 -> 91 us; the network on 8 patterns 1.08 -> 1.03 ms as a whole.
#pragma once
#include "cdx_unet_gemm.cuh"
#include "cdx_umma.cuh"

namespace cdx {
namespace unet {

constexpr int kCuTH = 16, kCuTW = 8;      // tile grid rows and columns of a CTA
constexpr int kCuThreads = 320;
constexpr int kCuSmem = 214 * 1024;       // dynamic shared memory a CTA may take
constexpr int kCuStagesMax = 8, kCuPatchMax = 3;
constexpr int kCuEpi = 20;                // floats a pixel's 16 channels take in the epilogue's staging (padded)

struct ConvUmma {
  const __nv_bfloat16 *x0, *x1;           // input parts (channels [0, C0) and [C0, C))
  const __nv_bfloat16* w;                 // packed weights [taps * C / 8][N][8]
  float *out0, *out1;                     // output channels [0, N0) and [N0, N)
  int C0, C, N0, N;
  int acc0, acc1;                         // add into the output
  int nimg, H, W;                         // input images
  int GH, GW, OH, OW;                     // tile grid and output image (the grid times out_s)
  int in_s, in_o, out_s;                  // patch origin: grid position * in_s + in_o
  int ph, pw;                             // patch rows and columns
  int split, pitch, par;                  // slot = split ? (x & 1) par + y pitch + x / 2 : y pitch + x
  int slots;                              // slots of a plane (odd: a pixel's planes fall on different banks)
  int sbo;                                // slots from one grid row to the next
  int ncls;                               // output parity classes (1 or 4)
  int ntap[4];
  short aoff[4][9], tap[4][9];            // first slot and weight tap of each class's taps
  int npatch, nstage, cch;                // patch buffers, weight stages, channels per stage (0 stages: resident)
  unsigned magic;                         // ceil(65536 / pw)
};

// no-swizzle K-major operand: start, LBO (one 16-byte K column to the next), SBO (8-row groups), version 1
__device__ __forceinline__ uint64_t cu_desc(unsigned saddr, unsigned lbo, unsigned sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 |
         (uint64_t)1 << 46;
}
__device__ __forceinline__ void cu_bulk(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

__global__ void __launch_bounds__(kCuThreads, 3) k_conv_umma(const __grid_constant__ ConvUmma a, int* __restrict__ err) {
  using namespace umma;
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ __align__(8) uint64_t afull[kCuPatchMax], aempty[kCuPatchMax], wfull[kCuStagesMax], wempty[kCuStagesMax],
      tfull[2], tempty[2], done;
  __shared__ unsigned tmem_base;
  __shared__ volatile int abort_flag;
  __shared__ __align__(16) float epi[4 * 32 * kCuEpi];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int C8 = a.C >> 3, N = a.N;
  const unsigned plane = (unsigned)a.slots * 16, patch = plane * C8;
  const unsigned patches = smem_u32(sm), weights = patches + a.npatch * patch;
  const unsigned wcol = (unsigned)N * 16;                    // bytes of eight K rows of the packed weights
  const unsigned stage_bytes = wcol * (a.cch >> 3);
  const int tx = (a.GW + kCuTW - 1) / kCuTW, ty = (a.GH + kCuTH - 1) / kCuTH;
  const int tiles = a.nimg * ty * tx;
  int cols = 32;                                             // TMEM columns: two accumulators
  while (cols < 2 * N) cols *= 2;

  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < kCuPatchMax; ++i) { mbar_init(smem_u32(&afull[i]), 128); mbar_init(smem_u32(&aempty[i]), 1); }
    for (int i = 0; i < kCuStagesMax; ++i) { mbar_init(smem_u32(&wfull[i]), 1); mbar_init(smem_u32(&wempty[i]), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&tfull[i]), 1); mbar_init(smem_u32(&tempty[i]), 128); }
    mbar_init(smem_u32(&done), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  net_wait();   // the barriers and TMEM are set up behind the predecessor's tail
  const unsigned tmem = tmem_base;
  auto give_up = [&]() {
    abort_flag = 1;
    atomicExch(err, 1);
  };

  if (warp < 4) {
    // ------------------------------------------------------------ patches
    // thread: channel plane tid % C8 of the pixels tid / C8, + 128 / C8, ...
    const int per = 128 / C8, c8 = tid % C8, p0 = tid / C8, c = c8 * 8;
    const bool active = p0 < per;
    const __nv_bfloat16* src = c < a.C0 ? a.x0 + c : a.x1 + (c - a.C0);
    const int ch = c < a.C0 ? a.C0 : a.C - a.C0;
    const int npx = a.ph * a.pw, D = a.npatch > 2 ? 1 : 0;   // D: patches in flight beyond the one signalled
    int g = 0;
    bool failed = false;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++g) {
      const int b = g % a.npatch, use = g / a.npatch;
      if (use > 0 && !mbar_wait_or_abort(smem_u32(&aempty[b]), (unsigned)((use - 1) & 1), &abort_flag)) {
        failed = true;
        break;
      }
      const int img = t / (ty * tx), r = t - img * ty * tx, y0 = r / tx * kCuTH * a.in_s + a.in_o,
                x0 = (r % tx) * kCuTW * a.in_s + a.in_o;
      const unsigned dst = patches + b * patch + c8 * plane;
      const __nv_bfloat16* base = src + (long long)img * a.H * a.W * ch;
      if (active)
        for (int p = p0; p < npx; p += per) {
          const int py = (int)((unsigned)p * a.magic >> 16), px = p - py * a.pw, y = y0 + py, x = x0 + px;
          const bool ok = y >= 0 && y < a.H && x >= 0 && x < a.W;
          const int slot = a.split ? (px & 1) * a.par + py * a.pitch + (px >> 1) : py * a.pitch + px;
          umma::cp16(dst + slot * 16, ok ? (const void*)(base + ((long long)y * a.W + x) * ch) : (const void*)a.w, ok);
        }
      cp_commit();
      if (D == 0) cp_wait<0>();
      else cp_wait<1>();
      if (g >= D) {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        mbar_arrive(smem_u32(&afull[(g - D) % a.npatch]));
      }
    }
    cp_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    if (failed) {
      give_up();
    } else if (D == 1 && g > 0) {
      mbar_arrive(smem_u32(&afull[(g - 1) % a.npatch]));
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------ epilogue
    // a warp's 32 grid pixels are four rows of eight; 16 channels at a time go through
    // shared memory so that four lanes write the 64 bytes of a pixel (a lane writing its
    // own pixel's 16-byte pieces left half sectors: 32 -> 32 at 256^2 x32, 161 -> 113 us)
    const int ew = warp - 4;
    float* tr = epi + ew * 32 * kCuEpi;
    int q = 0;
    bool failed = false;
    for (int t = blockIdx.x; t < tiles && !failed; t += gridDim.x) {
      const int img = t / (ty * tx), r = t - img * ty * tx;
      const int gy = r / tx * kCuTH + ew * 4, gx = (r % tx) * kCuTW + (lane >> 2);
      for (int cls = 0; cls < a.ncls; ++cls, ++q) {
        const int b = q & 1;
        if (!warp_wait_or_abort(smem_u32(&tfull[b]), (unsigned)((q >> 1) & 1), &abort_flag)) {
          if (lane == 0) give_up();
          failed = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const long long px = ((long long)img * a.OH + gy * a.out_s + (cls >> 1)) * a.OW + gx * a.out_s + (cls & 1);
        for (int c0 = 0; c0 < N; c0 += 16) {
          uint32_t v[16];
          const unsigned ta = tmem + ((unsigned)(ew * 32) << 16) + (unsigned)(b * N + c0);
          __syncwarp();   // the previous channels have been read, by lanes outside the grid too
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
              : "r"(ta)
              : "memory");
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
          for (int k = 0; k < 4; ++k)
            *reinterpret_cast<uint4*>(tr + lane * kCuEpi + 4 * k) = make_uint4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
          __syncwarp();
          const bool second = c0 >= a.N0, add = second ? a.acc1 : a.acc0;
          const int ch = second ? N - a.N0 : a.N0, c = (second ? c0 - a.N0 : c0) + 4 * (lane & 3);
          float* out = (second ? a.out1 : a.out0) + px * ch + c;
          const long long step = (long long)a.out_s * a.OW * ch;   // one grid row
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (gy + k >= a.GH || gx >= a.GW) continue;
            float4 f = *reinterpret_cast<const float4*>(tr + (8 * k + (lane >> 2)) * kCuEpi + 4 * (lane & 3));
            float4* o = reinterpret_cast<float4*>(out + k * step);
            if (add) {
              const float4 e = *o;
              f = make_float4(e.x + f.x, e.y + f.y, e.z + f.z, e.w + f.w);
            }
            *o = f;
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        mbar_arrive(smem_u32(&tempty[b]));
      }
    }
  } else if (warp == 8) {
    // ------------------------------------------------------------ MMA lane
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16(128, N);
      const int spc = a.cch >> 4, chunks = a.nstage ? (a.C + a.cch - 1) / a.cch : 1;
      const unsigned sbo = (unsigned)a.sbo * 16;
      bool failed = a.nstage == 0 && !mbar_wait_or_abort(smem_u32(&wfull[0]), 0, &abort_flag);
      int g = 0, q = 0, s = 0;
      unsigned sp = 0;   // weight stage and its phase
      for (int t = blockIdx.x; t < tiles && !failed; t += gridDim.x, ++g) {
        const int b = g % a.npatch;
        if (!mbar_wait_or_abort(smem_u32(&afull[b]), (unsigned)((g / a.npatch) & 1), &abort_flag)) {
          failed = true;
          break;
        }
        const unsigned pa = patches + b * patch;
        for (int cls = 0; cls < a.ncls && !failed; ++cls, ++q) {
          const int ab = q & 1;
          if (q >= 2 && !mbar_wait_or_abort(smem_u32(&tempty[ab]), (unsigned)(((q >> 1) - 1) & 1), &abort_flag)) {
            failed = true;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const unsigned d = tmem + (unsigned)(ab * N);
          // a 16-byte step of an operand's start is one more in its descriptor
          const uint64_t da = cu_desc(pa, plane, sbo);
          const unsigned as = 2 * plane >> 4, ws = 2 * wcol >> 4;
          if (a.nstage == 0) {
            const uint64_t dw = cu_desc(weights, wcol, 128);
            const int steps = a.C >> 4;
#pragma unroll 3
            for (int i = 0; i < a.ntap[cls]; ++i) {
              const uint64_t di = da + a.aoff[cls][i], dt = dw + (unsigned)a.tap[cls][i] * steps * ws;
#pragma unroll 2
              for (int kk = 0; kk < steps; ++kk) mma_f16(d, di + kk * as, dt + kk * ws, idesc, i > 0 || kk > 0);
            }
          } else {
            for (int i = 0; i < a.ntap[cls] && !failed; ++i) {
              const uint64_t di = da + a.aoff[cls][i];
              for (int k = 0; k < chunks; ++k) {
                if (!mbar_wait_or_abort(smem_u32(&wfull[s]), sp, &abort_flag)) {
                  failed = true;
                  break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint64_t dw = cu_desc(weights + s * stage_bytes, wcol, 128), dk = di + k * spc * as;
                const int steps = min(spc, (a.C >> 4) - k * spc);
#pragma unroll 8
                for (int kk = 0; kk < steps; ++kk) mma_f16(d, dk + kk * as, dw + kk * ws, idesc, i > 0 || k > 0 || kk > 0);
                mma_commit(smem_u32(&wempty[s]));
                if (++s == a.nstage) { s = 0; sp ^= 1; }
              }
            }
          }
          if (!failed) mma_commit(smem_u32(&tfull[ab]));
        }
        if (!failed) mma_commit(smem_u32(&aempty[b]));
      }
      if (failed) give_up();
      mma_commit(smem_u32(&done));   // arrives when every MMA this lane issued is complete
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ weight copies
    if (lane == 0) {
      if (a.nstage == 0) {
        int taps = 0;
        for (int cls = 0; cls < a.ncls; ++cls)
          for (int i = 0; i < a.ntap[cls]; ++i) taps = max(taps, a.tap[cls][i] + 1);
        cu_bulk(weights, a.w, (unsigned)taps * C8 * wcol, smem_u32(&wfull[0]));
        if (!mbar_wait(smem_u32(&wfull[0]), 0)) give_up();   // in place (or given up) before the CTA may end
      } else {
        const int chunks = (a.C + a.cch - 1) / a.cch;
        int s = 0;
        unsigned sp = 0;
        long long n = 0;
        bool failed = false;
        for (int t = blockIdx.x; t < tiles && !failed; t += gridDim.x)
          for (int cls = 0; cls < a.ncls && !failed; ++cls)
            for (int i = 0; i < a.ntap[cls] && !failed; ++i)
              for (int k = 0; k < chunks; ++k, ++n) {
                if (n >= a.nstage && !mbar_wait_or_abort(smem_u32(&wempty[s]), sp ^ 1, &abort_flag)) {
                  failed = true;
                  break;
                }
                const int col = a.tap[cls][i] * C8 + k * (a.cch >> 3), cnt = min(a.cch >> 3, C8 - k * (a.cch >> 3));
                cu_bulk(weights + s * stage_bytes, a.w + (long long)col * N * 8, cnt * wcol, smem_u32(&wfull[s]));
                if (++s == a.nstage) { s = 0; sp ^= 1; }
              }
        if (failed) {
          give_up();
          // the copies still in flight land before the CTA ends
          for (long long m = n < a.nstage ? 0 : n - a.nstage; m < n; ++m)
            if (!mbar_wait(smem_u32(&wfull[m % a.nstage]), (unsigned)((m / a.nstage) & 1))) break;
        }
      }
    }
    __syncwarp();
  }
  // TMEM is freed after the last MMA has completed and the epilogue's reads are done
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 8) {
    if (!warp_wait(smem_u32(&done), 0) && lane == 0) atomicExch(err, 1);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(cols) : "memory");
  }
}

// Shared-memory plan of a launch; false: the layer does not fit this kernel.
// Whole 16-channel K steps, parts and outputs that split on 16 channels, at most 32
// planes of channels (128 copy threads take 4 pixels at a time there), N <= 256 (two
// accumulators in 512 TMEM columns), and one patch plus two weight stages in kCuSmem.
inline bool cu_plan(ConvUmma& a, int taps, int& smem) {
  if (a.C % 16 || a.C0 % 16 || a.N % 16 || a.N0 % 16 || a.C > 256 || a.N > 256 || a.C < 16) return false;
  const int patch = a.slots * 2 * a.C, wall = taps * a.C * a.N * 2;
  a.magic = (65536 + a.pw - 1) / a.pw;
  if (wall + 2 * patch <= kCuSmem * 3 / 4) {   // resident weights, and room for copies in flight
    a.nstage = 0;
    a.cch = a.C;
    a.npatch = wall + 3 * patch <= 100 * 1024 ? 3 : 2;   // two CTAs per SM either way where they fit
    smem = a.npatch * patch + wall;
    return true;
  }
  a.cch = a.C;   // stages of about 16 KB: smaller ones spend the MMA lane on barriers
  while (a.cch % 32 == 0 && a.cch * a.N * 2 > 16384) a.cch /= 2;
  const int stage = a.cch * a.N * 2;
  a.npatch = 2 * patch + 2 * stage <= kCuSmem ? 2 : 1;
  a.nstage = std::min(kCuStagesMax, (kCuSmem - a.npatch * patch) / stage);
  smem = a.npatch * patch + a.nstage * stage;
  return a.nstage >= 2;
}

inline cudaError_t launch_conv_umma(const ConvUmma& a, int smem, int* err, bool dep, cudaStream_t st) {
  static std::atomic<unsigned long long> done{0};   // attribute set, bit per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (!(done.load(std::memory_order_acquire) & bit)) {
    if ((e = cudaFuncSetAttribute(k_conv_umma, cudaFuncAttributeMaxDynamicSharedMemorySize, kCuSmem)) != cudaSuccess)
      return e;
    done.fetch_or(bit, std::memory_order_release);
  }
  int cols = 32;
  while (cols < 2 * a.N) cols *= 2;
  // resident CTAs per SM: shared memory (228 KB, 1 KB reserved per CTA), TMEM columns, threads
  const int per_sm = std::max(1, std::min({(228 * 1024) / (smem + 1024 + 11 * 1024), 512 / cols, 3}));
  const long long tiles = (long long)a.nimg * ((a.GH + kCuTH - 1) / kCuTH) * ((a.GW + kCuTW - 1) / kCuTW);
  const int grid = (int)std::min<long long>(tiles, (long long)per_sm * sm_count());
  return net_launch(dep, k_conv_umma, grid, kCuThreads, smem, st, a, err);
}

// Geometry of the five forms.  3x3 stride 1 (flip: the data gradient's taps run the other way).
inline void cu_conv3(ConvUmma& a, bool flip) {
  a.in_s = a.out_s = 1;
  a.in_o = -1;
  a.ph = kCuTH + 2;
  a.pw = a.pitch = kCuTW + 2;
  a.split = a.par = 0;
  a.slots = a.ph * a.pitch + 1;
  a.sbo = a.pitch;
  a.ncls = 1;
  a.ntap[0] = 9;
  for (int k = 0; k < 9; ++k) {
    const int ky = k / 3, kx = k % 3;
    a.tap[0][k] = (short)k;
    a.aoff[0][k] = (short)(flip ? (2 - ky) * a.pitch + 2 - kx : ky * a.pitch + kx);
  }
}
// k x k stride 2, padding p (3x3 down convolution; 2x2: a transposed convolution's data gradient)
inline void cu_conv_s2(ConvUmma& a, int k, int p) {
  a.in_s = 2;
  a.out_s = 1;
  a.in_o = -p;
  a.ph = 2 * kCuTH - 2 + k;
  a.pw = 2 * kCuTW - 2 + k;
  a.split = 1;
  a.pitch = (a.pw + 1) / 2;
  a.par = a.ph * a.pitch;
  a.slots = 2 * a.par + 1;
  a.sbo = 2 * a.pitch;
  a.ncls = 1;
  a.ntap[0] = k * k;
  for (int t = 0; t < k * k; ++t) {
    const int ky = t / k, kx = t % k;
    a.tap[0][t] = (short)t;
    a.aoff[0][t] = (short)((kx & 1) * a.par + ky * a.pitch + (kx >> 1));
  }
}
// the adjoint of a k x k stride-2 convolution, padding p: output pixel (2y + cy, 2x + cx) takes
// the taps with (cy + p - ky) and (cx + p - kx) even, from input pixel (y, x) + that half
inline void cu_adj_s2(ConvUmma& a, int k, int p) {
  a.in_s = 1;
  a.out_s = 2;
  a.in_o = 0;
  a.ph = kCuTH + (k > 2);
  a.pw = a.pitch = kCuTW + (k > 2);
  a.split = a.par = 0;
  a.slots = a.ph * a.pitch | 1;
  a.sbo = a.pitch;
  a.ncls = 4;
  for (int c = 0; c < 4; ++c) {
    int n = 0;
    for (int t = 0; t < k * k; ++t) {
      const int dy = (c >> 1) + p - t / k, dx = (c & 1) + p - t % k;
      if (dy % 2 || dx % 2) continue;
      a.tap[c][n] = (short)t;
      a.aoff[c][n++] = (short)(dy / 2 * a.pitch + dx / 2);
    }
    a.ntap[c] = n;
  }
}

// ------------------------------------------------------------------- wgrad
// dW[co][tap][ci] = sum over output pixels m of dY[m][co] X[m at tap][ci].  Both
// operands are the channel planes above with the pixels as K (MN-major: a core matrix
// is eight pixels of eight channels), so one row segment of X serves the KW taps of a
// filter row at shifted starts.  A CTA takes one filter row, up to 128 channels of one
// side as M and up to 128 of the other as N (KW accumulators of N columns), and one
// split of the pixels, which it walks in order in steps of 16, as k_conv_wgrad does:
// the partial sums are the same, bit for bit.  Rows of M and columns of N past the
// channels multiply whatever lies behind the planes and are not read back.
// Bound by the chain of MMAs of a CTA (a split's pixels in order) and by the lane that
// issues them.  Batch 32 of 256^2: the step's 15 launches 8.5 -> 3.9 ms, and 2.9 with
// descriptors added to and the loop unrolled (32 -> 32 channels at 256^2 576 -> 350 us, the
// 1x1 head 306 -> 138; unrolled by 4 and by 8 1-2 % apart).
constexpr int kWgStages = 4, kWgAhead = 2;
constexpr int kWgThreads = 160;     // warps 0-3 copy and then drain the accumulators, warp 4 issues the MMAs

struct WgradUmma {
  const __nv_bfloat16 *x0, *x1, *dy;   // X parts (channels [0, C0) and [C0, Cin)), dY
  float* part;                         // [splits][Cout][KH * KW * Cin]
  int C0, Cin, Cout, H, W, Ho, Wo, KH, KW, S, P;
  int M, m_per_split;                  // output pixels, per split
  int m_is_x;                          // M side: X's channels (else dY's)
  int mt, nt, nn;                      // M tiles, N tiles, channels of an N tile
  int xslots, yslots, xpl, ypl;        // slots of a plane and planes of a stage, X and dY
  int seg;                             // output pixels of a stage (of one row)
  int stage, smem;                     // bytes of a stage, of the launch
};

// MN-major no-swizzle operand: SBO from eight channels to the next, LBO from eight pixels to the next
__device__ __forceinline__ uint64_t wg_desc(unsigned saddr, unsigned plane) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)(128 >> 4) << 16 | (uint64_t)(plane >> 4) << 32 |
         (uint64_t)1 << 46;
}

__global__ void __launch_bounds__(kWgThreads, 1) k_wgrad_umma(const __grid_constant__ WgradUmma a, int* __restrict__ err) {
  using namespace umma;
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ __align__(8) uint64_t full[kWgStages], empty[kWgStages], done;
  __shared__ unsigned tmem_base;
  __shared__ volatile int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ky = blockIdx.x % a.KH, mtile = blockIdx.x / a.KH % a.mt, ntile = blockIdx.x / a.KH / a.mt;
  const int mb = blockIdx.y * a.m_per_split, me = min(a.M, mb + a.m_per_split);
  const int cx0 = (a.m_is_x ? mtile * 128 : ntile * a.nn), cy0 = (a.m_is_x ? ntile * a.nn : mtile * 128);
  const int nx = min(a.m_is_x ? 128 : a.nn, a.Cin - cx0), ny = min(a.m_is_x ? a.nn : 128, a.Cout - cy0);
  const unsigned xplane = (unsigned)a.xslots * 16, yplane = (unsigned)a.yslots * 16;
  const int ncol = (a.nn + 15) & ~15;                       // columns of an accumulator
  int cols = 32;
  while (cols < a.KW * ncol) cols *= 2;

  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < kWgStages; ++i) { mbar_init(smem_u32(&full[i]), 128); mbar_init(smem_u32(&empty[i]), 1); }
    mbar_init(smem_u32(&done), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const unsigned tmem = tmem_base, base = smem_u32(sm);
  auto give_up = [&]() {
    abort_flag = 1;
    atomicExch(err, 1);
  };
  const int hw = a.Ho * a.Wo, par = a.seg + (a.KW > 1);    // slots of one column parity (stride 2)

  if (warp < 4) {
    // ------------------------------------------------------------ copies
    const int xp = nx / 8, yp = ny / 8, xper = 128 / xp, yper = 128 / yp;
    const int xc = tid % xp, xi = tid / xp, yc = tid % yp, yi = tid / yp;
    const int c = cx0 + xc * 8, ch = c < a.C0 ? a.C0 : a.Cin - a.C0;
    const __nv_bfloat16* xsrc = c < a.C0 ? a.x0 + c : a.x1 + (c - a.C0);
    const __nv_bfloat16* ysrc = a.dy + cy0 + yc * 8;
    int g = 0;
    bool failed = false;
    for (int m = mb; m < me && !failed; ++g) {
      const int s = g % kWgStages, use = g / kWgStages;
      if (use > 0 && !mbar_wait_or_abort(smem_u32(&empty[s]), (unsigned)((use - 1) & 1), &abort_flag)) {
        failed = true;
        break;
      }
      const int img = m / hw, r = m - img * hw, oy = r / a.Wo, ox = r - oy * a.Wo;
      const int len = min(min(a.seg, a.Wo - ox), me - m);
      const unsigned xd = base + s * a.stage + xc * xplane, yd = base + s * a.stage + a.xpl * xplane + yc * yplane;
      const int y = oy * a.S - a.P + ky, x0 = ox * a.S - a.P, npx = (len - 1) * a.S + a.KW;
      const bool row = y >= 0 && y < a.H;
      const __nv_bfloat16* xrow = xsrc + ((long long)img * a.H + (row ? y : 0)) * a.W * ch;
      if (xi < xper)
        for (int p = xi; p < npx; p += xper) {
          const int x = x0 + p, slot = a.S == 1 ? p : (p & 1) * par + (p >> 1);
          const bool ok = row && x >= 0 && x < a.W;
          umma::cp16(xd + slot * 16, ok ? (const void*)(xrow + (long long)x * ch) : (const void*)a.dy, ok);
        }
      if (yi < yper)
        for (int p = yi; p < len; p += yper) umma::cp16(yd + p * 16, ysrc + (long long)(m + p) * a.Cout, true);
      umma::cp_commit();
      if (g >= kWgAhead) {
        umma::cp_wait<kWgAhead>();
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        mbar_arrive(smem_u32(&full[(g - kWgAhead) % kWgStages]));
      }
      m += len;
    }
    umma::cp_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    if (failed) {
      give_up();
    } else {
      for (int q = g > kWgAhead ? g - kWgAhead : 0; q < g; ++q) mbar_arrive(smem_u32(&full[q % kWgStages]));
    }
    // ------------------------------------------------------------ partial sums
    if (!__all_sync(0xffffffffu, mbar_wait_or_abort(smem_u32(&done), 0, &abort_flag) && !abort_flag)) {
      if (lane == 0) give_up();
    } else {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int K = a.KH * a.KW * a.Cin, row = warp * 32 + lane, nm = a.m_is_x ? nx : ny, nv = a.m_is_x ? ny : nx;
      float* part = a.part + (long long)blockIdx.y * a.Cout * K;
      for (int t = 0; t < a.KW; ++t)
        for (int c0 = 0; c0 < ncol; c0 += 16) {
          uint32_t v[16];
          const unsigned ta = tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(t * ncol + c0);
          __syncwarp();   // lanes past the channels skip the stores
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
              : "r"(ta)
              : "memory");
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
          if (row >= nm) continue;
          const int k = (ky * a.KW + t) * a.Cin + cx0;
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (c0 + j < nv) {
              const float f = mb < me ? __uint_as_float(v[j]) : 0.f;
              if (a.m_is_x) part[(long long)(cy0 + c0 + j) * K + k + row] = f;
              else part[(long long)(cy0 + row) * K + k + c0 + j] = f;
            }
        }
    }
  } else {
    // ------------------------------------------------------------ MMA lane
    if (lane == 0) {
      // A and B MN-major (bits 15, 16)
      const uint32_t idesc = idesc_bf16(128, ncol) | (1u << 15) | (1u << 16);
      int g = 0;
      bool failed = false;
      for (int m = mb; m < me; ++g) {
        const int s = g % kWgStages, ox = m % a.Wo, len = min(min(a.seg, a.Wo - ox), me - m);
        if (!mbar_wait_or_abort(smem_u32(&full[s]), (unsigned)((g / kWgStages) & 1), &abort_flag)) {
          failed = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const unsigned xa = base + s * a.stage, ya = xa + a.xpl * xplane;
        const uint64_t dx = wg_desc(xa, xplane), dy = wg_desc(ya, yplane);   // a slot further is one more
        auto steps = [&](auto kw) {
          constexpr int KW = decltype(kw)::value;
          const uint64_t dm = a.m_is_x ? dx : dy, dn = a.m_is_x ? dy : dx;
#pragma unroll 8
          for (int p = 0; p < len; p += 16)
#pragma unroll
            for (int t = 0; t < KW; ++t) {
              const int off = a.S == 1 ? t : (t & 1) * par + (t >> 1);
              mma_f16(tmem + t * ncol, dm + p + (a.m_is_x ? off : 0), dn + p + (a.m_is_x ? 0 : off), idesc, g > 0 || p > 0);
            }
        };
        if (a.KW == 3) steps(std::integral_constant<int, 3>());
        else if (a.KW == 2) steps(std::integral_constant<int, 2>());
        else steps(std::integral_constant<int, 1>());
        mma_commit(smem_u32(&empty[s]));
        m += len;
      }
      if (failed) give_up();
      mma_commit(smem_u32(&done));
    }
    __syncwarp();
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 4) {
    if (!warp_wait(smem_u32(&done), 0) && lane == 0) atomicExch(err, 1);
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(cols) : "memory");
  }
}

// Tiles and shared memory of a launch over `splits` splits; false: the layer does not fit
// (16 output pixels of a K step have to lie in one row, whole 8-channel planes).
inline bool wg_plan(WgradUmma& a, int splits, int sms) {
  if (a.Wo % 16 || a.Cin % 8 || a.Cout % 8 || a.C0 % 8 || a.KW > 3 || a.S > 2 || a.m_per_split % 16) return false;
  a.m_is_x = a.Cin >= a.Cout;   // the larger side fills M
  const int mc = a.m_is_x ? a.Cin : a.Cout, nc = a.m_is_x ? a.Cout : a.Cin;
  a.mt = (mc + 127) / 128;
  auto sized = [&](int nn, int seg) {
    a.nn = std::min(nc, nn);
    a.nt = (nc + a.nn - 1) / a.nn;
    a.seg = seg;
    a.xpl = std::min(a.m_is_x ? 128 : a.nn, a.Cin) / 8;
    a.ypl = std::min(a.m_is_x ? a.nn : 128, a.Cout) / 8;
    a.xslots = (a.S == 1 ? seg + a.KW - 1 : 2 * (seg + (a.KW > 1))) | 1;
    a.yslots = seg | 1;
    a.stage = (a.xpl * a.xslots + a.ypl * a.yslots) * 16;
    // behind the last stage: what the unused rows and columns read (16 planes of either side at most)
    a.smem = kWgStages * a.stage + 16 * std::max(a.xslots, a.yslots) * 16;
    return a.KH * a.mt * a.nt * splits <= sms ? kCuSmem : kCuSmem / 2 - 8 * 1024;   // one CTA per SM, or two
  };
  // 128 columns of N unless that leaves SMs without a CTA; the longest segments that fit
  for (int nn = nc > 64 && a.KH * a.mt * ((nc + 127) / 128) * splits < sms ? 64 : 128; nn >= 64; nn -= 64)
    for (int seg = 256; seg >= 64; seg /= 2)
      if (a.Wo % seg == 0 || seg == 64) {
        const int budget = sized(nn, seg);
        if (a.smem <= (seg == 64 ? kCuSmem : budget)) return true;
      }
  return false;
}

inline cudaError_t launch_wgrad_umma(const WgradUmma& a, int splits, int* err, cudaStream_t st) {
  static std::atomic<unsigned long long> done{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (!(done.load(std::memory_order_acquire) & bit)) {
    if ((e = cudaFuncSetAttribute(k_wgrad_umma, cudaFuncAttributeMaxDynamicSharedMemorySize, kCuSmem)) != cudaSuccess)
      return e;
    done.fetch_or(bit, std::memory_order_release);
  }
  k_wgrad_umma<<<dim3(a.KH * a.mt * a.nt, splits), kWgThreads, a.smem, st>>>(a, err);
  return cudaGetLastError();
}

}  // namespace unet
}  // namespace cdx
