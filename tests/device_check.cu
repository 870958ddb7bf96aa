// Checks of device functions and internal entry points that no call of the C ABI reaches by
// itself.  Built and run by test_gpu_device_check.py against libgb300_bem.so:
//   device_check <check> [arguments]
// prints one line of figures; 1 is returned (with a message) if a CUDA call fails.
#include <algorithm>
#include <cmath>
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

__global__ void sincos_kernel(const double* r, const double* k, int n, const double2* trig, double2* out) {
  __shared__ double2 tab[kSincosTable];
  load_sincos_table(tab, trig);
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s, c;
  sincos_table(r[i], angle_units(k[i]), tab, &s, &c);
  out[i] = make_double2(c, s);
}

// sincos: largest absolute errors with the host's table and with the one that the CTA computes,
// and the largest relative error of the sine up to half a unit, over k from 1e-3 to 1e4 and k r
// from 1e-12 to 6e6, at the midpoints between two units, at the quadrants' edges and beside both.
int sincos_errors() {
  std::mt19937_64 rng(11);
  std::uniform_real_distribution<double> u01(0.0, 1.0);
  std::vector<double> r, k;
  const double h = 2.0 * M_PI / kSincosUnits;
  for (double kk : {1e-3, 0.37, 3.66, 57.3, 366.0, 1e4}) {
    auto add = [&](double kr) {
      for (int d = -1; d <= 1; ++d) {
        double v = kr / kk;
        if (d) v = std::nextafter(v, d < 0 ? 0.0 : 1e300);
        if (v * kk < 6.5e6) {
          r.push_back(v);
          k.push_back(kk);
        }
      }
    };
    for (int i = 0; i < 4000; ++i) add(std::pow(10.0, -12.0 + 18.8 * u01(rng)));
    for (int i = 0; i < 2000; ++i) add(700.0 * u01(rng));
    for (int i = 0; i < 1000; ++i) add((std::floor(i < 500 ? i : 2e9 * u01(rng)) + 0.5) * h);
    for (int i = 0; i < 600; ++i) add(0.5 * M_PI * (i < 300 ? i : std::floor(4e6 * u01(rng))));
  }
  r.push_back(0.0);
  k.push_back(3.66);
  const int n = (int)r.size();
  Dev<double> dr(r), dk(k);
  Dev<double2> dt(sincos_table_host()), out(n);
  double worst[2] = {0, 0}, small = 0;
  for (int t = 0; t < 2; ++t) {
    sincos_kernel<<<(n + 255) / 256, 256>>>(dr.p, dk.p, n, t ? nullptr : dt.p, out.p);
    ck(cudaGetLastError(), "sincos");
    ck(cudaDeviceSynchronize(), "sincos");
    const std::vector<double2> o = out.host();
    for (int i = 0; i < n; ++i) {
      // the exact angle as a double and its rounding error
      const double hi = k[i] * r[i], lo = std::fma(k[i], r[i], -hi);
      const long double sh = sinl(hi), ch = cosl(hi), sl = sinl(lo), cl = cosl(lo);
      const long double s = sh * cl + ch * sl, c = ch * cl - sh * sl;
      worst[t] = std::max(worst[t], (double)std::max(fabsl(o[i].y - s), fabsl(o[i].x - c)));
      if (hi > 0.0 && hi < 0.499 * h) small = std::max(small, (double)fabsl((o[i].y - s) / s));
    }
  }
  std::printf("%d %.3e %.3e %.3e\n", n, worst[0], worst[1], small);
  return 0;
}

// Kernels that a capture of `launch` holds.
template <typename F> int captured_kernels(F launch) {
  cudaStream_t stream;
  cudaGraph_t graph;
  ck(cudaStreamCreate(&stream), "stream");
  ck(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal), "begin capture");
  ck(launch(stream), "captured launch");
  ck(cudaStreamEndCapture(stream, &graph), "end capture");
  size_t n = 0;
  ck(cudaGraphGetNodes(graph, nullptr, &n), "nodes");
  std::vector<cudaGraphNode_t> nodes(n);
  ck(cudaGraphGetNodes(graph, nodes.data(), &n), "nodes");
  int kernels = 0;
  for (cudaGraphNode_t node : nodes) {
    cudaGraphNodeType type;
    ck(cudaGraphNodeGetType(node, &type), "node type");
    kernels += type == cudaGraphNodeTypeKernel;
  }
  ck(cudaGraphDestroy(graph), "destroy graph");
  ck(cudaStreamDestroy(stream), "destroy stream");
  return kernels;
}

// launch_counts: calls whose reported number of launches is not what they launch, of the
// right-hand side (excitations 1..4) and the regular pairs, both forms, 1..64 frequencies.  The
// launches are captured, not run; every pointer is a zeroed buffer all the same.
int launch_counts() {
  Dev<char> zeros(std::vector<char>((size_t)64 << 20));
  void* z = zeros.p;
  bem::DeviceMesh m;
  m.faces32 = (bem::FaceF32*)z;
  m.faces64 = (bem::FaceF64*)z;
  m.lane_slots = (bem::LaneSlot*)z;
  m.group_faces32 = (float*)z;
  m.tile_group_ptr = m.tile_row_base = m.col_ptr = m.col_fb = m.vertex_row = m.driven = (int*)z;
  m.pairs_by_test_ptr = m.pairs_by_test = (int*)z;
  m.pairs = (bem::SingularPair*)z;
  m.trig = (double2*)z;
  m.nv = 8;
  m.nf = 12;
  m.Q = 6;
  m.n_tiles = 1;
  m.max_tile_rows = 40;
  m.ntr = 1;
  std::vector<double> k(64);
  std::vector<bem::OperatorCoeffs> c(64);
  std::vector<double2> q(64, make_double2(0.0, 1.0)), cD(64, make_double2(1.0, 0.0)), cH(64);
  for (int i = 0; i < 64; ++i) {
    k[i] = 1.0 + i;
    cH[i] = make_double2(0.0, -1.0 / k[i]);
  }
  int wrong = 0, calls = 0;
  for (bem::Precision prec : {bem::Precision::Mixed, bem::Precision::FP64})
    for (int n = 1; n <= 64; ++n) {
      for (int nc = 1; nc <= 4; ++nc, ++calls)
        wrong += bem::rhs_launches(prec, nc, n) != captured_kernels([&](cudaStream_t s) {
          return bem::launch_rhs_freqs(m, prec, n, k.data(), c.data(), q.data(), z, nc, z, 12, z, z, 32, s);
        });
      ++calls;
      wrong += bem::regular_launches(m, prec, n) != captured_kernels([&](cudaStream_t s) {
        return bem::launch_regular(m, prec, n, k.data(), cD.data(), cH.data(), z, 64, 4096, s);
      });
    }
  std::printf("%d %d\n", calls, wrong);
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  auto is = [&](const char* name, int args) { return argc == args + 2 && std::strcmp(argv[1], name) == 0; };
  if (is("block_inverse", 2)) return block_inverse(std::atoi(argv[2]), std::atoi(argv[3]));
  if (is("launch_counts", 0)) return launch_counts();
  if (is("sincos", 0)) return sincos_errors();
  std::printf("unknown check\n");
  return 1;
}
