// A pipeline wait that ran out is reported by the call it happened in, once: the word the
// kernels set is set here from the host.  Built with the library's own objects; needs a GPU.
#include "cdx_unet.cu"

#include <cstdio>

int main() {
  cdx_unet_config c;
  cdx_unet_config_default(&c);
  c.n = 32;
  c.levels = 2;
  c.base = 16;
  c.batch = 1;
  cdx_unet* u = nullptr;
  if (cdx_unet_create(&c, nullptr, &u)) return std::printf("create: %s\n", last_error()), 2;
  const int P = c.n * c.n;
  float *in = nullptr, *out = nullptr;
  if (cudaMalloc(&in, sizeof(float) * P) || cudaMalloc(&out, sizeof(float) * 4 * P)) return 2;
  std::vector<float> h(P), a(4 * P), b(4 * P);
  for (int i = 0; i < P; ++i) h[i] = (float)(i % 37);
  cudaMemcpy(in, h.data(), sizeof(float) * P, cudaMemcpyHostToDevice);
  bool ok = true;
  auto expect = [&](const char* what, bool good) {
    std::printf("%s: %s\n", what, good ? "ok" : "FAILED");
    ok = ok && good;
  };
  auto forward = [&](std::vector<float>& v) {
    const int e = cdx_unet_forward(u, in, out, 1);
    cudaDeviceSynchronize();
    cudaMemcpy(v.data(), out, sizeof(float) * 4 * P, cudaMemcpyDeviceToHost);
    return e;
  };
  auto set_word = [&]() {
    const int one = 1;
    return cudaMemcpy(u->net.umma_err, &one, sizeof one, cudaMemcpyHostToDevice);
  };
  double loss = 0.0;
  auto backward = [&]() { return cdx_unet_loss_backward(u, in, in, in, in, 1, &loss); };
  expect("a pass", forward(a) == CDX_OK && set_word() == cudaSuccess);
  expect("the pass that finds the word set", forward(b) == CDX_ERR_CUDA);
  expect("the pass after it", forward(b) == CDX_OK && std::memcmp(a.data(), b.data(), sizeof(float) * 4 * P) == 0);
  expect("a training pass that finds it set", set_word() == cudaSuccess && backward() == CDX_ERR_CUDA);
  expect("the training pass after it", backward() == CDX_OK);
  cdx_unet_destroy(u);
  cudaFree(in);
  cudaFree(out);
  std::printf(ok ? "error word ok\n" : "error word FAILED\n");
  return ok ? 0 : 1;
}
