// Exterior field evaluation (sm_103a).
//
// u(x) = sum over source points y_s of [dG/dn_y(x, y_s) p(y_s) - G(x, y_s) q_s] w_s
// with the sources at the regular quadrature points of every face, p
// interpolated with the P1 basis and q the DP0 Neumann data: the reference's
// evaluate_galerkin_field_cpu (src/blab/solvers/julia_local/src/
// BeatEngineCpuField.jl:1-45) over build_field_evaluation_cache
// (BeatEngineCore.jl:1240-1280, symmetry off).  The reference's CUDA version
// uses one block per observation point with an FP32 shared-memory reduction
// (BeatEngineCudaField.jl:102-189).
//
// Here: a prologue kernel forms the weighted sources p_s w_s (all frequencies
// and excitations of a batch), then the FP32 kernel runs one cluster per (32
// observation points, up to four frequencies), its CTAs sharing out the faces,
// and the FP64 kernel one CTA per (observation point, frequency).  The mixed form uses the same compensated
// phase as the assembly (double-float k|c_g - x| per face, FP32 correction per
// point), compensated FP32 partial sums per thread and an FP64 block
// reduction; the far field sits at kr ~ 500 rad at 16 kHz, where plain FP32
// phase would lose ~3e-5 rad.
#include <cooperative_groups.h>

#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>

#include "bem_common.cuh"
#include "bem_kernels.h"

namespace cg = cooperative_groups;

namespace bem {
namespace {

// Rule weights w_q and basis values phi_a(xi_q) (a-major), passed by value.
template <typename R> struct FieldRule {
  R w[kMaxQ];
  R phi[3 * kMaxQ];
};

// sources[((bt*nc + c)*nf + g)*Q + q] = 2A_g w_q sum_a phi_a(xi_q) p[bt][c][v(g,a)]
template <typename R>
__global__ void field_sources_kernel(const int* __restrict__ faces, const double* __restrict__ area, int nf, int Q,
                                     int nc, const typename cplx<R>::type* __restrict__ p, long long ldp,
                                     typename cplx<R>::type* __restrict__ src, int total, FieldRule<R> fr) {
  typedef typename cplx<R>::type C2;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int q = i % Q;
  const int g = (i / Q) % nf;
  const int bc = i / (Q * nf);  // bt*nc + c
  const C2* pv = p + (size_t)bc * ldp;
  const R w = fr.w[q], phi0 = fr.phi[q], phi1 = fr.phi[Q + q], phi2 = fr.phi[2 * Q + q];
  const C2 a = pv[faces[3 * g]], b = pv[faces[3 * g + 1]], c = pv[faces[3 * g + 2]];
  const R s = (R)(2.0 * area[g]) * w;
  C2 v;
  v.x = (phi0 * a.x + phi1 * b.x + phi2 * c.x) * s;
  v.y = (phi0 * a.y + phi1 * b.y + phi2 * c.y) * s;
  src[i] = v;
}

struct FieldParamsF32 {
  df kdf[64];
  float k[64];
  float2 qscale[64];
};

// Adds x to the running sum s; the rounding error of the addition, which two_sum gives
// exactly, goes to c, so s + c carries the terms' sum to about 2^-44.
__device__ __forceinline__ void comp_add(float& s, float& c, float x) {
  const df t = two_sum(s, x);
  s = t.hi;
  c += t.lo;
}

// One cluster per (32 observation points, NFQ frequencies starting at NFQ * blockIdx.y):
// lane = observation point; the cluster's CTAs and their eight warps take the faces in
// turn (face g goes to warp g mod (8 CTAs of the cluster)).  Every lane of a warp works on
// the same face, so face records, sources and drives are broadcast loads, and everything
// that does not depend on the frequency is formed once per (point, face) or (point,
// source): the double-float distance |c_g - x|, s = 2 C.d + d.d, 1/r,
// the compensated r - |C| = s / (r + |C|) and the normal-derivative factor.  Per frequency
// remain the reduction of k|C| mod 2 pi, the phase, e^{ikr} and
//   fs += e^{ikr} [ (t/r)(ik - 1/r) p_s w_s - q w_s / r ] / (4 pi).
// The Q terms of a face are summed in FP32 and added to a compensated per-lane sum
// (comp_add: exact rounding errors, so the split of the faces over warps and CTAs moves
// the result by about 1e-13 only); the warps' and then the CTAs' sums are added in
// FP64 in a fixed order, the latter through distributed shared memory, so the split needs
// no workspace.  Frequencies of the last group beyond the batch are computed on the
// batch's last frequency and not stored.
//
// Bound: FP32 issue where the grid fills the GPU.  Before the faces were shared out over a
// cluster, a call of one frequency ran one CTA per 32 points, each warp sweeping an eighth
// of all the faces: 68 CTAs on 152 SMs for 2,146 points and 9,948 faces (2.0 ms; now
// 0.4 ms), 5 CTAs for 146 points and 1,036 faces (0.22 ms; now 0.06 ms).
constexpr int kFieldWarps = 8;
constexpr int kFieldMaxSplit = 8;

template <int Q, int NC, int NFQ>
__global__ void __launch_bounds__(256) field_f32_kernel(const FaceF32* __restrict__ faces, int nf,
                                                        const float2* __restrict__ src,
                                                        const float2* __restrict__ drive,  // NC x nf
                                                        const double* __restrict__ obs, int nobs,
                                                        const FieldParamsF32* __restrict__ prm, int batch,
                                                        double2* __restrict__ out, FieldRule<float> fr, int ntr,
                                                        int4 trs) {
  cg::cluster_group cluster = cg::this_cluster();
  const int split = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int o = (blockIdx.x / split) * 32 + lane;
  const int f0 = blockIdx.y * NFQ;
  const bool live = o < nobs;
  const int oc = live ? o : nobs - 1;  // idle lanes repeat a live point; their result is dropped
  const double xo[3] = {obs[3 * oc], obs[3 * oc + 1], obs[3 * oc + 2]};
  float xhi[3], xlo[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    xhi[d] = (float)xo[d];
    xlo[d] = (float)(xo[d] - (double)xhi[d]);
  }
  int bt[NFQ];
  df kdf[NFQ];
  float k[NFQ];
  float2 qs[NFQ];
#pragma unroll
  for (int f = 0; f < NFQ; ++f) {
    bt[f] = min(f0 + f, batch - 1);
    kdf[f] = prm->kdf[bt[f]];
    k[f] = prm->k[bt[f]];
    qs[f] = prm->qscale[bt[f]];
  }
  float ar[NFQ][NC], ac[NFQ][NC], br[NFQ][NC], bcmp[NFQ][NC];
#pragma unroll
  for (int f = 0; f < NFQ; ++f)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      ar[f][c] = 0.f;
      ac[f][c] = 0.f;
      br[f][c] = 0.f;
      bcmp[f][c] = 0.f;
    }
  // sources: every face and, under symmetry, its images (BeatEngineCore.jl:1240-1280)
  for (int ti = 0; ti < ntr; ++ti)
  for (int g = rank * kFieldWarps + wid; g < nf; g += split * kFieldWarps) {
    const FaceF32& F = faces[g];
    const int tr = ti == 0 ? trs.x : ti == 1 ? trs.y : ti == 2 ? trs.z : trs.w;
    const float sg[3] = {(tr & 1) ? -1.f : 1.f, (tr & 2) ? -1.f : 1.f, 1.f};
    const float nrm[3] = {sg[0] * F.normal[0], sg[1] * F.normal[1], F.normal[2]};
    df C[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      df s = two_sum(sg[d] * F.anchor_hi[d], -xhi[d]);
      s.lo += sg[d] * F.anchor_lo[d] - xlo[d];
      C[d] = quick_two_sum(s.hi, s.lo);
    }
    const df R2 = df_add(df_add(df_mul(C[0], C[0]), df_mul(C[1], C[1])), df_mul(C[2], C[2]));
    const df R = df_sqrt(R2);
    const float R0 = R.hi + R.lo;
    float theta0[NFQ];
#pragma unroll
    for (int f = 0; f < NFQ; ++f) theta0[f] = df_reduce_two_pi(df_mul(kdf[f], R));
    const float Cf[3] = {C[0].hi + C[0].lo, C[1].hi + C[1].lo, C[2].hi + C[2].lo};
    const float C2[3] = {2.f * Cf[0], 2.f * Cf[1], 2.f * Cf[2]};
    const float Cn = fmaf(Cf[0], nrm[0], fmaf(Cf[1], nrm[1], Cf[2] * nrm[2]));
    float2 qg[NFQ][NC], fs[NFQ][NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float2 dr = drive[(size_t)c * nf + g];
#pragma unroll
      for (int f = 0; f < NFQ; ++f) {
        // every rounding spelled out: the same bits whichever NFQ a frequency runs in
        qg[f][c] = make_float2(__fmul_rn(fmaf(qs[f].x, dr.x, -__fmul_rn(qs[f].y, dr.y)), F.area2),
                               __fmul_rn(fmaf(qs[f].x, dr.y, __fmul_rn(qs[f].y, dr.x)), F.area2));
        fs[f][c] = make_float2(0.f, 0.f);
      }
    }
#pragma unroll
    for (int n = 0; n < Q; ++n) {
      const float d[3] = {sg[0] * F.off[3 * n], sg[1] * F.off[3 * n + 1], F.off[3 * n + 2]};
      const float dd = fmaf(d[0], d[0], fmaf(d[1], d[1], d[2] * d[2]));
      const float s = fmaf(C2[0], d[0], fmaf(C2[1], d[1], fmaf(C2[2], d[2], dd)));
      const float rv[3] = {Cf[0] + d[0], Cf[1] + d[1], Cf[2] + d[2]};
      const float rr = fmaf(rv[0], rv[0], fmaf(rv[1], rv[1], rv[2] * rv[2]));  // not |C|^2 + s: that cancels close by
      const float rinv = rr > 1e-30f ? rsqrt_ftz(rr) : 0.f;
      const float r = rr * rinv;
      const float delta = s * rcp_ftz(fmaxf(r + R0, 1e-30f));
      const float sc = rinv * BEM_INV_FOUR_PI;
      // (r . n_y) / r with r . n_y = C . n + d . n (d . n = 0 for points on the face plane, kept for generality)
      const float t = (Cn + fmaf(d[0], nrm[0], fmaf(d[1], nrm[1], d[2] * nrm[2]))) * rinv * sc;
      const float nta = -t * rinv;          // -(t/r)/r / (4 pi)
      const float nscw = -sc * fr.w[n];     // -w/r / (4 pi)
#pragma unroll
      for (int f = 0; f < NFQ; ++f) {
        const float th = reduce_two_pi(fmaf(k[f], delta, theta0[f]));
        float sn, cs;
        sincos_ftz(th, &sn, &cs);
        const float tb = t * k[f];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const float2 ps = src[(((size_t)bt[f] * NC + c) * nf + g) * Q + n];
          const float zx = fmaf(nta, ps.x, fmaf(-tb, ps.y, nscw * qg[f][c].x));
          const float zy = fmaf(nta, ps.y, fmaf(tb, ps.x, nscw * qg[f][c].y));
          fs[f][c].x = fmaf(cs, zx, fmaf(-sn, zy, fs[f][c].x));
          fs[f][c].y = fmaf(cs, zy, fmaf(sn, zx, fs[f][c].y));
        }
      }
    }
#pragma unroll
    for (int f = 0; f < NFQ; ++f)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        comp_add(ar[f][c], ac[f][c], fs[f][c].x);
        comp_add(br[f][c], bcmp[f][c], fs[f][c].y);
      }
  }
  __shared__ double2 red[kFieldWarps][NC][32];
  __shared__ double2 tot[NFQ][NC][32];  // this CTA's sums, read by the cluster's first CTA
#pragma unroll
  for (int f = 0; f < NFQ; ++f) {
#pragma unroll
    for (int c = 0; c < NC; ++c)
      red[wid][c][lane] =
          make_double2((double)ar[f][c] + (double)ac[f][c], (double)br[f][c] + (double)bcmp[f][c]);
    __syncthreads();
    if (wid < NC) {
      double vr = 0.0, vi = 0.0;
      for (int w = 0; w < kFieldWarps; ++w) {
        vr += red[w][wid][lane].x;
        vi += red[w][wid][lane].y;
      }
      tot[f][wid][lane] = make_double2(vr, vi);
    }
    __syncthreads();
  }
  if (split > 1) cluster.sync();
  if (rank == 0 && wid < NFQ * NC && live) {  // NFQ x NC <= 4 warps, one (frequency, excitation) each
    const int f = wid / NC, c = wid - f * NC;
    if (f0 + f < batch) {
      double vr = 0.0, vi = 0.0;
      for (int r = 0; r < split; ++r) {
        const double2 v = *cluster.map_shared_rank(&tot[f][c][lane], r);
        vr += v.x;
        vi += v.y;
      }
      out[((size_t)(f0 + f) * NC + c) * nobs + o] = make_double2(vr, vi);
    }
  }
  if (split > 1) cluster.sync();  // no CTA leaves while the first may still read its sums
}

// Clusters of `split` CTAs of a field kernel that are resident at once (asked of the driver
// once per device, kernel and size).
int resident_clusters(const void* kern, int split) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int>, int> known;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  auto it = known.find({dev, kern, split});
  if (it != known.end()) return it->second;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(split);
  cfg.blockDim = dim3(kFieldWarps * 32);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    n = std::max(1, 2 * sm_count() / split);
  }
  known[{dev, kern, split}] = n;
  return n;
}

// CTAs of a cluster that share the faces of 32 points.  The time goes as (waves of clusters)
// / split: 157 clusters of four, one wave and a bit, took 0.88 ms where the sevens' two full
// waves take 0.67 (5,000 points, 9,948 faces, three-point rule).  A warp keeps at least
// four faces.
int field_split(const void* kern, long long clusters, int nf) {
  int best = 1;
  double best_time = 1e300;
  for (int s = 1; s <= kFieldMaxSplit && (s == 1 || nf >= s * kFieldWarps * 4); ++s) {
    const long long cap = resident_clusters(kern, s);
    const double time = (double)((clusters + cap - 1) / cap) / s;
    if (time < 0.999 * best_time) {
      best = s;
      best_time = time;
    }
  }
  return best;
}

template <typename K, typename... A>
cudaError_t launch_field_f32(K kern, unsigned pt_blocks, unsigned groups, unsigned rule_groups, int nf,
                             cudaStream_t stream, A... args) {
  const int split = field_split((const void*)kern, (long long)pt_blocks * rule_groups, nf);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(pt_blocks * split, groups);
  cfg.blockDim = dim3(kFieldWarps * 32);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

struct FieldParamsF64 {
  double k[64];
  double2 qscale[64];
};

// A CTA per observation point and NFQ frequencies, its threads over the faces.  Bound by the
// FP64 pipe: 23 instructions of geometry per point and source, 22 per frequency; up to four
// frequencies share the geometry (1,000 points, 1,280 triangles, 16 frequencies:
// 10.5 -> 7.0 ms; two at 3,984: 4.35 -> 3.41).
template <int Q, int NC, int NFQ>
__global__ void __launch_bounds__(256) field_f64_kernel(const FaceF64* __restrict__ faces, int nf,
                                                        const double2* __restrict__ src,
                                                        const double2* __restrict__ drive,
                                                        const double* __restrict__ obs, int nobs,
                                                        const FieldParamsF64* __restrict__ prm, int batch,
                                                        double2* __restrict__ out, FieldRule<double> fr, int ntr,
                                                        int4 trs, const double2* __restrict__ trig) {
  __shared__ double2 tab[kSincosTable];
  load_sincos_table(tab, trig);
  __syncthreads();
  const int o = blockIdx.x, f0 = blockIdx.y * NFQ;
  const double xo[3] = {obs[3 * o], obs[3 * o + 1], obs[3 * o + 2]};
  double kf[NFQ];
  AngleUnits ku[NFQ];
  double2 acc[NFQ][NC];
#pragma unroll
  for (int f = 0; f < NFQ; ++f) {  // a frequency beyond the batch repeats the last one
    kf[f] = prm->k[min(f0 + f, batch - 1)];
    ku[f] = angle_units(kf[f]);
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[f][c] = make_double2(0., 0.);
  }
  for (int ti = 0; ti < ntr; ++ti)  // every face and its symmetry images
  for (int g = threadIdx.x; g < nf; g += blockDim.x) {
    const FaceF64& F = faces[g];
    const int tr = ti == 0 ? trs.x : ti == 1 ? trs.y : ti == 2 ? trs.z : trs.w;
    const double sg[3] = {(tr & 1) ? -1.0 : 1.0, (tr & 2) ? -1.0 : 1.0, 1.0};
    double2 qg[NFQ][NC];
#pragma unroll
    for (int f = 0; f < NFQ; ++f)
#pragma unroll
      for (int c = 0; c < NC; ++c)
        qg[f][c] = cscale(cmul(prm->qscale[min(f0 + f, batch - 1)], drive[(size_t)c * nf + g]), F.area2);
#pragma unroll
    for (int n = 0; n < Q; ++n) {
      double rv[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) rv[d] = (sg[d] * F.anchor[d] - xo[d]) + sg[d] * F.off[3 * n + d];
      const double rr = rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2];
      if (is_zero(rr)) continue;
      const double rinv = rsqrt(rr), r = rr * rinv;
      const double sc = rinv * (0.25 / CUDART_PI);
      // e^{ikr} [ (t/r)(ik - 1/r) p_s w_s - q w_s / r ] / (4 pi), t = (r . n_y) / r
      const double t = (rv[0] * sg[0] * F.normal[0] + rv[1] * sg[1] * F.normal[1] + rv[2] * F.normal[2]) * rinv * sc;
      const double nta = -t * rinv, nscw = -sc * fr.w[n];
#pragma unroll
      for (int f = 0; f < NFQ; ++f) {
        double sn, cs;
        sincos_table(r, ku[f], tab, &sn, &cs);
        const double tb = t * kf[f];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const double2 ps = src[(((size_t)min(f0 + f, batch - 1) * NC + c) * nf + g) * Q + n];
          const double zx = fma(nta, ps.x, fma(-tb, ps.y, nscw * qg[f][c].x));
          const double zy = fma(nta, ps.y, fma(tb, ps.x, nscw * qg[f][c].y));
          acc[f][c].x = fma(cs, zx, fma(-sn, zy, acc[f][c].x));
          acc[f][c].y = fma(cs, zy, fma(sn, zx, acc[f][c].y));
        }
      }
    }
  }
  __shared__ double red[2 * NFQ * NC][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int f = 0; f < NFQ; ++f)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      double vr = acc[f][c].x, vi = acc[f][c].y;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        vr += __shfl_xor_sync(0xffffffffu, vr, s);
        vi += __shfl_xor_sync(0xffffffffu, vi, s);
      }
      if (lane == 0) {
        red[2 * (f * NC + c)][wid] = vr;
        red[2 * (f * NC + c) + 1][wid] = vi;
      }
    }
  __syncthreads();
  if (threadIdx.x < NFQ * NC && f0 + (int)threadIdx.x / NC < batch) {
    const int fc = threadIdx.x;
    double vr = 0, vi = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      vr += red[2 * fc][w];
      vi += red[2 * fc + 1][w];
    }
    out[((size_t)f0 * NC + fc) * nobs + o] = make_double2(vr, vi);
  }
}

}  // namespace

static df host_df(double x) {
  df r;
  r.hi = (float)x;
  r.lo = (float)(x - (double)r.hi);
  return r;
}

cudaError_t launch_field(const DeviceMesh& m, Precision prec, int batch, const double* k, const double2* qscale,
                         const void* pressure, long long ldp, int nc, const void* drive, const double* obs, int nobs,
                         void* sources, double2* out, cudaStream_t stream, int rule_batch) {
  if (rule_batch <= 0) rule_batch = batch;
  if (batch > 64 || nc < 1 || nc > 4 || nobs <= 0) return cudaErrorInvalidValue;
  FieldRule<float> fr32;
  FieldRule<double> fr64;
  for (int i = 0; i < kMaxQ; ++i) {
    fr32.w[i] = (float)m.rule_w[i];
    fr64.w[i] = m.rule_w[i];
  }
  for (int i = 0; i < 3 * kMaxQ; ++i) {
    fr32.phi[i] = (float)m.rule_phi[i];
    fr64.phi[i] = m.rule_phi[i];
  }
  const int total = batch * nc * m.nf * m.Q;
  if (prec == Precision::Mixed) {
    field_sources_kernel<float><<<(total + 255) / 256, 256, 0, stream>>>(m.faces, m.area, m.nf, m.Q, nc,
                                                                         (const float2*)pressure, ldp,
                                                                         (float2*)sources, total, fr32);
    FieldParamsF32 hp;
    for (int b = 0; b < batch; ++b) {
      hp.kdf[b] = host_df(k[b]);
      hp.k[b] = (float)k[b];
      hp.qscale[b] = make_float2((float)qscale[b].x, (float)qscale[b].y);
    }
    FieldParamsF32* dp = (FieldParamsF32*)((char*)sources + (((size_t)total * sizeof(float2) + 255) / 256) * 256);
    cudaMemcpyAsync(dp, &hp, sizeof(hp), cudaMemcpyHostToDevice, stream);
    // NFQ frequencies per cluster share the frequency-independent geometry: the largest of
    // four, two and one with NFQ x nc <= 4 (the sums stay in registers) that the batch fills
    int nfq = 1;
    for (int cand = 4; cand >= 2; cand /= 2)
      if (cand * nc <= 4 && cand <= batch) {
        nfq = cand;
        break;
      }
    const unsigned pt_blocks = (unsigned)((nobs + 31) / 32);
    const int4 trs = make_int4(m.tr[0], m.tr[1], m.tr[2], m.tr[3]);
    cudaError_t le = cudaSuccess;
    auto run = [&](auto kern, int per_cluster) {
      le = launch_field_f32(kern, pt_blocks, (unsigned)((batch + per_cluster - 1) / per_cluster),
                            (unsigned)((rule_batch + per_cluster - 1) / per_cluster), m.nf, stream,
                            (const FaceF32*)m.faces32, m.nf, (const float2*)sources, (const float2*)drive, obs, nobs,
                            (const FieldParamsF32*)dp, batch, out, fr32, m.ntr, trs);
    };
#define BEM_F32(QQ, NCC, NFQQ) run(field_f32_kernel<QQ, NCC, NFQQ>, NFQQ)
#define BEM_F32_Q(NCC, NFQQ) \
  if (m.Q == 6)              \
    BEM_F32(6, NCC, NFQQ);   \
  else if (m.Q == 3)         \
    BEM_F32(3, NCC, NFQQ);   \
  else                       \
    BEM_F32(1, NCC, NFQQ);
    if (nc == 1 && nfq == 4) {
      BEM_F32_Q(1, 4)
    } else if (nc == 1 && nfq == 2) {
      BEM_F32_Q(1, 2)
    } else if (nc == 2 && nfq == 2) {
      BEM_F32_Q(2, 2)
    } else {
      switch (nc) {
        case 1: BEM_F32_Q(1, 1) break;
        case 2: BEM_F32_Q(2, 1) break;
        case 3: BEM_F32_Q(3, 1) break;
        default: BEM_F32_Q(4, 1) break;
      }
    }
#undef BEM_F32_Q
#undef BEM_F32
    if (le != cudaSuccess) return le;
  } else {
    field_sources_kernel<double><<<(total + 255) / 256, 256, 0, stream>>>(m.faces, m.area, m.nf, m.Q, nc,
                                                                          (const double2*)pressure, ldp,
                                                                          (double2*)sources, total, fr64);
    FieldParamsF64 hp;
    for (int b = 0; b < batch; ++b) {
      hp.k[b] = k[b];
      hp.qscale[b] = qscale[b];
    }
    FieldParamsF64* dp = (FieldParamsF64*)((char*)sources + (((size_t)total * sizeof(double2) + 255) / 256) * 256);
    cudaMemcpyAsync(dp, &hp, sizeof(hp), cudaMemcpyHostToDevice, stream);
    // frequencies per CTA by the instructions of a point and source: 23 of geometry and 22 per
    // frequency, a partly filled last group's included
    int nfq = 1, cost = 45 * batch;
    for (int cand = 2; cand * nc <= 4; cand *= 2)
      if (const int t = (batch + cand - 1) / cand * (23 + 22 * cand); t < cost) {
        nfq = cand;
        cost = t;
      }
    const dim3 grid64(nobs, (batch + nfq - 1) / nfq);
    const int4 trs = make_int4(m.tr[0], m.tr[1], m.tr[2], m.tr[3]);
    auto run = [&](auto kern) {
      kern<<<grid64, 256, 0, stream>>>(m.faces64, m.nf, (const double2*)sources, (const double2*)drive, obs, nobs, dp,
                                       batch, out, fr64, m.ntr, trs, m.trig);
    };
    auto run_q = [&](auto nc_c, auto nfq_c) {
      constexpr int NC = decltype(nc_c)::value, NFQ = decltype(nfq_c)::value;
      if (m.Q == 6)
        run(field_f64_kernel<6, NC, NFQ>);
      else if (m.Q == 3)
        run(field_f64_kernel<3, NC, NFQ>);
      else
        run(field_f64_kernel<1, NC, NFQ>);
    };
    using One = std::integral_constant<int, 1>;
    using Two = std::integral_constant<int, 2>;
    if (nc == 1 && nfq == 4)
      run_q(One{}, std::integral_constant<int, 4>{});
    else if (nc == 1 && nfq == 2)
      run_q(One{}, Two{});
    else if (nc == 2 && nfq == 2)
      run_q(Two{}, Two{});
    else if (nc == 1)
      run_q(One{}, One{});
    else if (nc == 2)
      run_q(Two{}, One{});
    else if (nc == 3)
      run_q(std::integral_constant<int, 3>{}, One{});
    else
      run_q(std::integral_constant<int, 4>{}, One{});
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Single-excitation, single-frequency field evaluation from caller-placed
// buffers (face records, weighted sources, drive, parameter block).  Used by
// the allocation-free entry point in bem_noalloc.cu; the parameter block is
// written on the device by write_field_params so no host staging is needed.
namespace {
__global__ void write_field_params_f32(FieldParamsF32* prm, double k) {
  df v;
  v.hi = (float)k;
  v.lo = (float)(k - (double)v.hi);
  prm->kdf[0] = v;
  prm->k[0] = (float)k;
  prm->qscale[0] = make_float2(1.0f, 0.0f);
}
__global__ void write_field_params_f64(FieldParamsF64* prm, double k) {
  prm->k[0] = k;
  prm->qscale[0] = make_double2(1.0, 0.0);
}
}  // namespace

size_t field_params_bytes() { return sizeof(FieldParamsF32) > sizeof(FieldParamsF64) ? sizeof(FieldParamsF32) : sizeof(FieldParamsF64); }

cudaError_t launch_field_single(Precision prec, const void* faces, int nf, int Q, const double* rule_w,
                                const double* rule_phi, const void* sources, const void* drive, const double* obs,
                                int nobs, double k, void* params, double2* out, cudaStream_t stream) {
  FieldRule<float> fr32;
  FieldRule<double> fr64;
  for (int i = 0; i < kMaxQ; ++i) {
    fr32.w[i] = (float)rule_w[i];
    fr64.w[i] = rule_w[i];
  }
  for (int i = 0; i < 3 * kMaxQ; ++i) {
    fr32.phi[i] = (float)rule_phi[i];
    fr64.phi[i] = rule_phi[i];
  }
  dim3 grid(nobs, 1);
  if (prec == Precision::Mixed) {
    FieldParamsF32* dp = (FieldParamsF32*)params;
    write_field_params_f32<<<1, 1, 0, stream>>>(dp, k);
    const FaceF32* f = (const FaceF32*)faces;
    const float2* s = (const float2*)sources;
    const float2* d = (const float2*)drive;
    auto run = [&](auto kern) {
      return launch_field_f32(kern, (unsigned)((nobs + 31) / 32), 1u, 1u, nf, stream, f, nf, s, d, obs, nobs,
                              (const FieldParamsF32*)dp, 1, out, fr32, 1, make_int4(0, 0, 0, 0));
    };
    const cudaError_t le = Q == 6   ? run(field_f32_kernel<6, 1, 1>)
                           : Q == 3 ? run(field_f32_kernel<3, 1, 1>)
                                    : run(field_f32_kernel<1, 1, 1>);
    if (le != cudaSuccess) return le;
  } else {
    FieldParamsF64* dp = (FieldParamsF64*)params;
    write_field_params_f64<<<1, 1, 0, stream>>>(dp, k);
    const FaceF64* f = (const FaceF64*)faces;
    const double2* s = (const double2*)sources;
    const double2* d = (const double2*)drive;
    if (Q == 6)
      field_f64_kernel<6, 1, 1><<<grid, 256, 0, stream>>>(f, nf, s, d, obs, nobs, dp, 1, out, fr64, 1, make_int4(0, 0, 0, 0),
                                                     nullptr);
    else if (Q == 3)
      field_f64_kernel<3, 1, 1><<<grid, 256, 0, stream>>>(f, nf, s, d, obs, nobs, dp, 1, out, fr64, 1, make_int4(0, 0, 0, 0),
                                                     nullptr);
    else
      field_f64_kernel<1, 1, 1><<<grid, 256, 0, stream>>>(f, nf, s, d, obs, nobs, dp, 1, out, fr64, 1, make_int4(0, 0, 0, 0),
                                                     nullptr);
  }
  return cudaGetLastError();
}

}  // namespace bem
