// Checks of device functions and internal entry points that no call of the C ABI reaches by
// itself.  Built and run by test_gpu_device_check.py against libgb300_bem.so:
//   device_check <check> [arguments]
// prints one line of figures; 1 is returned (with a message) if a CUDA call fails.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "bem_common.cuh"
#include "bem_kernels.h"

namespace {

void ck(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return;
  std::printf("%s: %s\n", what, cudaGetErrorString(e));
  std::exit(1);
}

template <typename T> struct Dev {
  T* p = nullptr;
  size_t n;
  explicit Dev(size_t n_) : n(n_) { ck(cudaMalloc(&p, n * sizeof(T)), "cudaMalloc"); }
  explicit Dev(const std::vector<T>& h) : Dev(h.size()) {
    ck(cudaMemcpy(p, h.data(), n * sizeof(T), cudaMemcpyHostToDevice), "to device");
  }
  ~Dev() { cudaFree(p); }
  std::vector<T> host() const {
    std::vector<T> h(n);
    ck(cudaMemcpy(h.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost), "to host");
    return h;
  }
};

// Factors of order n: unit lower with small multipliers, upper scaled by 2^e.
std::vector<float2> factors(int n, long long lda, int batch, int e, unsigned seed) {
  std::mt19937 rng(seed);
  std::uniform_real_distribution<float> u(-0.1f, 0.1f);
  std::vector<float2> a((size_t)lda * n * batch, make_float2(0.f, 0.f));
  for (int b = 0; b < batch; ++b)
    for (int j = 0; j < n; ++j)
      for (int i = 0; i < n; ++i) {
        float2 v = make_float2(u(rng) + (i == j ? 1.f : 0.f), u(rng));
        if (i <= j) v = make_float2(std::ldexp(v.x, e), std::ldexp(v.y, e));
        a[((size_t)b * n + j) * lda + i] = v;
      }
  return a;
}

// block_inverse n e: entries of the blocks' inverses that differ, to the bit, from those of the
// same factors unscaled (the upper side's times 2^-e), and entries that are not finite.
int block_inverse(int n, int e) {
  const long long lda = (n + 31) / 32 * 32;
  const size_t count = bem::lu_inverse_bytes(n, 1) / sizeof(float2);
  std::vector<float2> out[2];
  for (int k = 0; k < 2; ++k) {
    Dev<float2> a(factors(n, lda, 1, k ? e : 0, 7)), inv(count);
    ck(bem::lu_block_inverses(a.p, lda, n, 1, inv.p, 0), "block inverses");
    ck(cudaDeviceSynchronize(), "block inverses");
    out[k] = inv.host();
  }
  long long differ = 0, bad = 0;
  const size_t block = (size_t)bem::kOuterBlock * bem::kOuterBlock;
  for (size_t i = 0; i < count; ++i) {
    const bool upper = (i / block) % 2 == 1;
    const float2 x = out[0][i], y = out[1][i];
    const int s = upper ? -e : 0;
    differ += std::ldexp(x.x, s) != y.x || std::ldexp(x.y, s) != y.y;
    bad += !std::isfinite(x.x) || !std::isfinite(x.y) || !std::isfinite(y.x) || !std::isfinite(y.y);
  }
  std::printf("%lld %lld\n", differ, bad);
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  auto is = [&](const char* name, int args) { return argc == args + 2 && std::strcmp(argv[1], name) == 0; };
  if (is("block_inverse", 2)) return block_inverse(std::atoi(argv[2]), std::atoi(argv[3]));
  std::printf("unknown check\n");
  return 1;
}
