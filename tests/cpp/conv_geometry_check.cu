// Host check of the patch geometry of k_conv_umma (cdx_unet_umma.cuh): for each form,
// every row a tap's operand reads is a slot the copy warps fill, with the input pixel
// the convolution (or its adjoint) takes there; each output pixel's taps are the ones
// that reach it; and the shared-memory plan stays within its limits.
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <map>
#include <set>
#include <utility>

#include "cdx_unet_umma.cuh"

using namespace cdx::unet;

static bool ok = true;
static void fail(const char* form, const char* what) {
  std::printf("%s: %s\n", form, what);
  ok = false;
}

// adj: the adjoint of the k x k convolution of stride s, padding p
static void check(const char* form, const ConvUmma& a, int k, int s, int p, bool adj) {
  std::map<int, std::pair<int, int>> filled;   // slot -> patch pixel
  const unsigned magic = (65536 + a.pw - 1) / a.pw;
  for (int i = 0; i < a.ph * a.pw; ++i) {
    const int py = (int)((unsigned)i * magic >> 16), px = i - py * a.pw;
    if (py != i / a.pw || px < 0 || px >= a.pw) fail(form, "patch division");
    const int slot = a.split ? (px & 1) * a.par + py * a.pitch + (px >> 1) : py * a.pitch + px;
    if (slot < 0 || slot >= a.slots || filled.count(slot)) fail(form, "slot");
    filled[slot] = {py, px};
  }
  const int ty = 3, tx = 5;   // any tile: its origin in the grid
  for (int cls = 0; cls < a.ncls; ++cls)
    for (int r = 0; r < 128; ++r) {
      const int gy = ty * kCuTH + (r >> 3), gx = tx * kCuTW + (r & 7);
      const int oy = gy * a.out_s + (cls >> 1), ox = gx * a.out_s + (cls & 1);
      std::set<int> taps;
      int last = -1;
      for (int i = 0; i < a.ntap[cls]; ++i) {
        const int t = a.tap[cls][i], ky = t / k, kx = t % k;
        if (t <= last) fail(form, "taps out of order");
        last = t;
        taps.insert(t);
        const auto it = filled.find(a.aoff[cls][i] + (r >> 3) * a.sbo + (r & 7));
        if (it == filled.end()) { fail(form, "a tap reads a slot that is not filled"); continue; }
        const int y = ty * kCuTH * a.in_s + a.in_o + it->second.first, x = tx * kCuTW * a.in_s + a.in_o + it->second.second;
        if (!adj) {
          if (y != oy * s - p + ky || x != ox * s - p + kx) fail(form, "input pixel");
        } else if (y * s != oy + p - ky || x * s != ox + p - kx) {
          fail(form, "adjoint input pixel");
        }
      }
      for (int t = 0; t < k * k; ++t) {
        const bool reaches = !adj || ((oy + p - t / k) % s == 0 && (ox + p - t % k) % s == 0);
        if (reaches != (taps.count(t) > 0)) fail(form, "taps of an output pixel");
      }
    }
  // plans over the channel counts the kernel takes
  for (int C = 16; C <= 256; C += 16)
    for (int N = 16; N <= 256; N += 16) {
      ConvUmma b = a;
      b.C = b.C0 = C;
      b.N = b.N0 = N;
      int smem = 0;
      if (!cu_plan(b, k * k, smem)) continue;
      const int patch = b.slots * 2 * C;
      const int need = b.npatch * patch + (b.nstage ? b.nstage * b.cch * N * 2 : k * k * C * N * 2);
      if (smem != need || smem > kCuSmem || b.npatch < 1 || b.npatch > kCuPatchMax || b.nstage > kCuStagesMax ||
          b.nstage == 1 || (b.nstage && b.cch % 16) || patch % 16 || b.slots >= 1 << 14)
        fail(form, "shared-memory plan");
      if (128 / (C / 8) < 1) fail(form, "copy threads");
    }
}

int main() {
  ConvUmma a{};
  cu_conv3(a, false); check("3x3", a, 3, 1, 1, false);
  cu_conv3(a, true); check("3x3 data gradient", a, 3, 1, 1, true);
  cu_conv_s2(a, 3, 1); check("3x3 stride 2", a, 3, 2, 1, false);
  cu_conv_s2(a, 2, 0); check("2x2 stride 2", a, 2, 2, 0, false);
  cu_adj_s2(a, 3, 1); check("3x3 stride 2 data gradient", a, 3, 2, 1, true);
  cu_adj_s2(a, 2, 0); check("2x2 transposed", a, 2, 2, 0, true);
  std::printf(ok ? "geometry ok\n" : "geometry FAILED\n");
  return ok ? 0 : 1;
}
