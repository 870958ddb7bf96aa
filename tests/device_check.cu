// Checks of device functions and internal entry points that no call of the C ABI reaches by
// itself.  Built and run by test_gpu_device_check.py against libgb300_bem.so:
//   device_check <check> [arguments]
// prints one line of figures; 1 is returned (with a message) if a CUDA call fails.
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "bem_common.cuh"
#include "bem_kernels.h"

namespace bem {
int regular_width_f64(const DeviceMesh& m);
}

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

// solves n nrhs: relative difference between the block solves and the cluster substitution that
// takes over where their rows do not fit, on the same FP32 factors and right-hand sides, and
// the larger of both residuals ||P b - L U x|| / (|| |L| |U| |x| ||) in double.
int solves(int n, int nrhs) {
  const int batch = 2;
  const long long lda = (n + 31) / 32 * 32, ldb = lda;
  std::vector<float2> a = factors(n, lda, batch, 0, 3);
  // a diagonal that dominates keeps the solutions of a random triangle bounded
  for (int b = 0; b < batch; ++b)
    for (int i = 0; i < n; ++i) a[((size_t)b * n + i) * lda + i].x += 3.f;
  for (auto& v : a) {
    v.x *= 2.f / std::sqrt((float)n);
    v.y *= 2.f / std::sqrt((float)n);
  }
  for (int b = 0; b < batch; ++b)
    for (int i = 0; i < n; ++i) a[((size_t)b * n + i) * lda + i].x += 1.f;
  std::vector<float2> rhs((size_t)batch * nrhs * ldb, make_float2(0.f, 0.f));
  std::mt19937 rng(5);
  std::uniform_real_distribution<float> u(-1.f, 1.f);
  std::vector<int> perm((size_t)batch * n);
  for (int b = 0; b < batch; ++b) {
    for (int i = 0; i < n; ++i) perm[(size_t)b * n + i] = i;
    std::shuffle(perm.begin() + (size_t)b * n, perm.begin() + (size_t)(b + 1) * n, rng);
    for (int c = 0; c < nrhs; ++c)
      for (int i = 0; i < n; ++i) rhs[((size_t)b * nrhs + c) * ldb + i] = make_float2(u(rng), u(rng));
  }
  Dev<float2> da(a), d1(rhs), d2(rhs), inv(bem::lu_inverse_bytes(n, batch) / sizeof(float2));
  Dev<int> dp(perm);
  ck(bem::lu_block_inverses(da.p, lda, n, batch, inv.p, 0), "block inverses");
  ck(bem::lu_solve_blocks_batched(da.p, lda, n, batch, inv.p, dp.p, d1.p, ldb, nrhs, 0), "block solves");
  ck(bem::lu_solve_cluster_batched(bem::Precision::Mixed, da.p, lda, n, batch, dp.p, d2.p, ldb, nrhs, 0), "cluster solves");
  ck(cudaDeviceSynchronize(), "solves");
  const std::vector<float2> x[2] = {d1.host(), d2.host()};
  double diff = 0, norm = 0, worst = 0;
  for (size_t i = 0; i < rhs.size(); ++i) {
    diff += std::pow((double)x[0][i].x - x[1][i].x, 2) + std::pow((double)x[0][i].y - x[1][i].y, 2);
    norm += std::pow((double)x[0][i].x, 2) + std::pow((double)x[0][i].y, 2);
  }
  using cd = std::complex<double>;
  for (int k = 0; k < 2; ++k)
    for (int s = 0; s < batch * nrhs; ++s) {
      const float2* M = a.data() + (size_t)(s / nrhs) * n * lda;
      std::vector<cd> y(n), z(n);
      std::vector<double> ya(n), za(n);
      auto at = [&](int i, int j) { return cd(M[(size_t)j * lda + i].x, M[(size_t)j * lda + i].y); };
      for (int j = 0; j < n; ++j) {  // y = U x
        const cd xv(x[k][(size_t)s * ldb + j].x, x[k][(size_t)s * ldb + j].y);
        for (int i = 0; i <= j; ++i) {
          y[i] += at(i, j) * xv;
          ya[i] += std::abs(at(i, j)) * std::abs(xv);
        }
      }
      for (int j = 0; j < n; ++j) {  // z = L y
        z[j] += y[j];
        za[j] += ya[j];
        for (int i = j + 1; i < n; ++i) {
          z[i] += at(i, j) * y[j];
          za[i] += std::abs(at(i, j)) * ya[j];
        }
      }
      double r = 0, scale = 0;
      for (int i = 0; i < n; ++i) {
        const float2 b = rhs[(size_t)s * ldb + perm[(size_t)(s / nrhs) * n + i]];
        r += std::norm(cd(b.x, b.y) - z[i]);
        scale += za[i] * za[i];
      }
      worst = std::max(worst, std::sqrt(r / scale));
    }
  std::printf("%.3e %.3e\n", std::sqrt(diff / norm), worst);
  return 0;
}

// Entries of small factors and right-hand sides by a hash of their index.
__global__ void fill_kernel(float2* a, long long count, long long lda, float scale, float diagonal) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  unsigned long long h = (unsigned long long)i * 0x9e3779b97f4a7c15ull + 12345;
  h ^= h >> 31;
  h *= 0xbf58476d1ce4e5b9ull;
  h ^= h >> 29;
  const float re = (float)(int)(unsigned)h * 0x1p-31f, im = (float)(int)(unsigned)(h >> 32) * 0x1p-31f;
  a[i] = make_float2(scale * re + (i / lda == i % lda ? diagonal : 0.f), scale * im);
}

// rhs_groups n nrhs: entries of the block solves of nrhs right-hand sides together that differ, to
// the bit, from each by itself, and entries that are not finite.
int rhs_groups(int n, int nrhs) {
  const long long lda = (n + 31) / 32 * 32, ldb = lda;
  std::vector<int> perm(n);
  for (int i = 0; i < n; ++i) perm[i] = n - 1 - i;
  Dev<float2> a((size_t)lda * n), b((size_t)ldb * nrhs), x((size_t)ldb * nrhs), inv(bem::lu_inverse_bytes(n, 1) / sizeof(float2));
  Dev<int> dp(perm);
  fill_kernel<<<(unsigned)((a.n + 255) / 256), 256>>>(a.p, (long long)a.n, lda, 0.5f / n, 1.f);
  fill_kernel<<<(unsigned)((b.n + 255) / 256), 256>>>(b.p, (long long)b.n, ldb, 1.f, 0.f);
  ck(bem::lu_block_inverses(a.p, lda, n, 1, inv.p, 0), "block inverses");
  ck(cudaMemcpy(x.p, b.p, b.n * sizeof(float2), cudaMemcpyDeviceToDevice), "copy");
  ck(bem::lu_solve_blocks_batched(a.p, lda, n, 1, inv.p, dp.p, x.p, ldb, nrhs, 0), "solves together");
  for (int c = 0; c < nrhs; ++c)
    ck(bem::lu_solve_blocks_batched(a.p, lda, n, 1, inv.p, dp.p, b.p + c * ldb, ldb, 1, 0), "solve by itself");
  ck(cudaDeviceSynchronize(), "solves");
  const std::vector<float2> together = x.host(), alone = b.host();
  long long differ = 0, bad = 0;
  for (int c = 0; c < nrhs; ++c)
    for (int i = 0; i < n; ++i) {
      const float2 u = together[c * ldb + i], v = alone[c * ldb + i];
      differ += u.x != v.x || u.y != v.y;
      bad += !std::isfinite(u.x) || !std::isfinite(u.y);
    }
  std::printf("%lld %lld\n", differ, bad);
  return 0;
}

// edges: whether the dispatch of the solves (orders) and of the FP64 regular kernel (tile rows)
// changes where the figures beside it say.
int edges() {
  auto width = [](int rows) {
    bem::DeviceMesh m;
    m.max_tile_rows = rows;
    return bem::regular_width_f64(m);
  };
  std::printf("%d %d %d %d %d %d\n", bem::lu_solve_blocks_fits(43264), bem::lu_solve_blocks_fits(43265), width(581),
              width(582), width(1162), width(1163));
  return 0;
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
  if (is("solves", 2)) return solves(std::atoi(argv[2]), std::atoi(argv[3]));
  if (is("rhs_groups", 2)) return rhs_groups(std::atoi(argv[2]), std::atoi(argv[3]));
  if (is("edges", 0)) return edges();
  if (is("launch_counts", 0)) return launch_counts();
  if (is("sincos", 0)) return sincos_errors();
  std::printf("unknown check\n");
  return 1;
}
