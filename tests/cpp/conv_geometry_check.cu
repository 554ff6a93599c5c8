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

// weight gradient: the slots of one stage (a row segment), and the shared-memory plan
static void check_wgrad(int KW, int S, int P) {
  WgradUmma a{};
  a.KH = a.KW = KW; a.S = S; a.P = P;
  a.m_per_split = 32;
  for (int Wo : {16, 64, 256})
  for (int splits : {1, 64})
  for (int Cin = 8; Cin <= 520; Cin += 8)
    for (int Cout = 8; Cout <= 520; Cout += 8) {
      a.Cin = a.C0 = Cin; a.Cout = Cout; a.Wo = Wo;
      if (!wg_plan(a, splits, 152)) { fail("wgrad", "a layer of whole 8s does not fit"); continue; }
      const int mc = a.m_is_x ? Cin : Cout, nc = a.m_is_x ? Cout : Cin, ncol = (a.nn + 15) & ~15;
      if (a.mt * 128 < mc || a.nt * a.nn < nc || KW * ncol > 512 || ncol > 256) fail("wgrad", "tiles");
      if (a.smem > kCuSmem || a.seg % 16) fail("wgrad", "shared-memory plan");
      // operands read 16 (M) and ncol / 8 (N) planes from the start of the last stage's halves
      const long long last = (long long)(kWgStages - 1) * a.stage;
      const int xr = a.m_is_x ? 16 : ncol / 8, yr = a.m_is_x ? ncol / 8 : 16;
      if (last + 16LL * xr * a.xslots > a.smem || last + 16LL * a.xpl * a.xslots + 16LL * yr * a.yslots > a.smem)
        fail("wgrad", "an operand ends past the shared memory");
      if (a.xpl * 8 < std::min(a.m_is_x ? 128 : a.nn, Cin) || a.ypl * 8 < std::min(a.m_is_x ? a.nn : 128, Cout))
        fail("wgrad", "planes");
    }
  for (int C = 8; C <= 128; C *= 4) {
  a.Cin = a.C0 = a.Cout = C; a.Wo = 256;
  if (!wg_plan(a, 64, 152)) fail("wgrad", "plan");
  const int par = a.seg + (KW > 1);
  for (int len = 16; len <= a.seg; len += 16) {
    std::map<int, int> filled;
    for (int p = 0; p < (len - 1) * S + KW; ++p) {
      const int slot = S == 1 ? p : (p & 1) * par + (p >> 1);
      if (slot >= a.xslots || filled.count(slot)) fail("wgrad", "slot");
      filled[slot] = p;
    }
    for (int p = 0; p < len; p += 16)
      for (int t = 0; t < KW; ++t)
        for (int i = 0; i < 16; ++i) {
          const int slot = (S == 1 ? p + t : (t & 1) * par + p + (t >> 1)) + i;
          if (!filled.count(slot) || filled[slot] != (p + i) * S + t) fail("wgrad", "tap pixel");
        }
    if (len > a.yslots) fail("wgrad", "dY slots");
  }
  }
}

int main() {
  check_wgrad(3, 1, 1); check_wgrad(3, 2, 1); check_wgrad(2, 2, 0); check_wgrad(1, 1, 0);
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
