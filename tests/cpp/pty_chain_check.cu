// The kernels of a scan position launched dependently (as a sweep does) and plainly give
// the same bits: many sweeps over windows that overlap almost wholly, on odd and even
// columns and over the object's edges, so that every window holds what the position
// before wrote.  Needs a GPU.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "cdx_ptycho.cuh"

using namespace cdx;

#define CK(x)                                                                \
  do {                                                                       \
    const cudaError_t e_ = (x);                                              \
    if (e_ != cudaSuccess) {                                                 \
      std::printf("%s: %s\n", #x, cudaGetErrorString(e_));                   \
      std::exit(2);                                                          \
    }                                                                        \
  } while (0)

__global__ void next_sweep(int* iter) { *iter += 1; }

static unsigned rng = 12345u;
static float uniform() {
  rng = rng * 1664525u + 1013904223u;
  return (float)(rng >> 8) / 16777216.f;
}
template <class V>
static V* upload(const std::vector<V>& h) {
  V* d = nullptr;
  CK(cudaMalloc(&d, sizeof(V) * h.size()));
  CK(cudaMemcpy(d, h.data(), sizeof(V) * h.size(), cudaMemcpyHostToDevice));
  return d;
}

template <int N>
static std::vector<float2> twiddles() {
  std::vector<float2> t(std::max(1, Geom<N>::TWN), make_float2(1.f, 0.f));
  for (int plan = 0; plan < 2; ++plan)
    for (int p = 1; p < plan_len(N); ++p) {
      const int R = plan_radix_x(N, plan, p), NS = plan_ns_x(N, plan, p);
      for (int r = 1; r < R; ++r)
        for (int k = 0; k < NS; ++k) {
          const double w = 2.0 * M_PI * r * k / ((double)R * NS);
          t[tw_offset_x(N, plan, p) + (r - 1) * NS + k] = make_float2((float)std::cos(w), (float)-std::sin(w));
        }
    }
  return t;
}

// object after `sweeps` sweeps
template <int N>
static std::vector<float2> run(bool dependent, int oc, int sweeps) {
  using G = FGeom<N>;
  rng = 12345u;
  const int orows = N + 9, ns = 7;
  const int cp = (N + G::L - 1) / G::L * G::L;
  std::vector<float2> obj((size_t)orows * oc), probe((size_t)N * N);
  for (auto& v : obj) v = make_float2(0.5f + uniform(), uniform() - 0.5f);
  for (auto& v : probe) v = make_float2(uniform(), uniform());
  std::vector<float> pats((size_t)ns * N * cp);
  for (auto& v : pats) v = uniform();
  std::vector<int2> win = {{1, 1}, {2, 3}, {0, 2}, {3, oc - N}, {-5, 5}, {4, -3}, {6, 4}};
  std::vector<int> order((size_t)sweeps * ns);
  for (int s = 0; s < sweeps; ++s)
    for (int k = 0; k < ns; ++k) order[s * ns + k] = (k * (1 + s % 6) + s) % ns;   // ns is prime
  const float scal[2] = {2.f, 2.f};
  PtyArgs a{};
  float2* o = upload(obj);
  a.obj = o;
  a.W = upload(std::vector<float2>((size_t)N * cp));
  a.probe = upload(probe);
  a.step = upload(std::vector<float2>((size_t)N * N));
  a.pats = upload(pats);
  a.order = upload(order);
  int* iter = upload(std::vector<int>(1, 0));
  a.iter = iter;
  a.win = upload(win);
  a.scal = upload(std::vector<float>(scal, scal + 2));
  a.tw = upload(twiddles<N>());
  int* err = upload(std::vector<int>(1, 0));
  a.err = err;
  a.pat_stride = (long long)N * cp;
  a.rows = a.cols = N;
  a.obj_rows = orows;
  a.obj_cols = oc;
  while ((1 << a.tl) < G::L) ++a.tl;
  a.nscan = ns;
  a.norm = 1.f / N;
  a.maximum = 0.95f;
  a.obj_step = 1.f;
  a.pss = 1.f / ns;
  CK(pty_prepare<N>());
  cudaStream_t st;
  CK(cudaStreamCreate(&st));
  const dim3 rows((N + G::L - 1) / G::L);
  constexpr int colsm = G::SMEM_LINES + 2 * G::L * N * (int)sizeof(float);
  for (int s = 0; s < sweeps; ++s) {
    for (a.k = 0; a.k < ns; ++a.k) {
      if (dependent) {
        CK(pty_launch_fwd<N>(a, st));
        CK(pty_launch_col<N>(a, st));
        CK(pty_launch_upd<N>(a, st));
      } else {
        pty_fwd_rk<N, false><<<rows, G::T, PtyRow<N>::SMEM, st>>>(a);
        pty_col_rk<N><<<rows, G::T, colsm, st>>>(a);
        pty_upd_rk<N, false><<<rows, G::T, PtyRow<N>::SMEM, st>>>(a);
      }
    }
    next_sweep<<<1, 1, 0, st>>>(iter);
  }
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(st));
  int e = 0;
  CK(cudaMemcpy(&e, err, sizeof e, cudaMemcpyDeviceToHost));
  if (e) std::printf("a staging copy timed out\n");
  CK(cudaMemcpy(obj.data(), o, sizeof(float2) * obj.size(), cudaMemcpyDeviceToHost));
  for (const void* p : {(const void*)a.obj, (const void*)a.W, (const void*)a.probe, (const void*)a.step, (const void*)a.pats,
                        (const void*)a.order, (const void*)iter, (const void*)a.win, (const void*)a.scal,
                        (const void*)a.tw, (const void*)err})
    CK(cudaFree((void*)p));
  CK(cudaStreamDestroy(st));
  return obj;
}

template <int N>
static bool check(int oc, int sweeps) {
  const std::vector<float2> d = run<N>(true, oc, sweeps), p = run<N>(false, oc, sweeps);
  size_t bad = 0;
  bool finite = true;
  for (size_t i = 0; i < d.size(); ++i) {
    bad += d[i].x != p[i].x || d[i].y != p[i].y;
    finite = finite && std::isfinite(p[i].x) && std::isfinite(p[i].y);
  }
  std::printf("N=%d object columns %d, %d sweeps: %zu of %zu pixels differ%s\n", N, oc, sweeps, bad, d.size(),
              finite ? "" : ", not finite");
  return bad == 0 && finite;
}

int main() {
  bool ok = true;
  for (int extra : {8, 9}) {   // even and odd object widths
    ok = check<48>(48 + extra, 200) && ok;
    ok = check<256>(256 + extra, 200) && ok;
    ok = check<1024>(1024 + extra, 20) && ok;
  }
  std::printf(ok ? "chain ok\n" : "chain FAILED\n");
  return ok ? 0 : 1;
}
