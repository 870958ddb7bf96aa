// Shared device helpers for the GB300 exterior Helmholtz BEM kernels.
//
// Complex numbers are interleaved (re, im) float2 / double2.  "df" is
// double-float arithmetic: a value carried as an unevaluated sum hi + lo of two
// floats, built from the error-free transformations two-sum (Knuth) and
// two-product (via fmaf).  It carries ~44 bits of significand at a handful of
// FP32 instructions per operation, which matters on this part: FP64 issues at a
// small fraction of the FP32 rate.
#pragma once

#include <cuda_runtime.h>
#include <math_constants.h>
#include <math.h>
#include <stdint.h>

#include <vector>

#define BEM_HD __host__ __device__ __forceinline__
#define BEM_D __device__ __forceinline__

// Programmatic dependent launch, for chains of short kernels: a kernel launched with
// launch_chained may start while its predecessor in the stream drains.  It calls grid_wait
// before its first access to memory that an earlier kernel writes or reads (the wait ends
// when all earlier grids are complete and their writes visible), and reads such memory with
// plain loads, never through the read-only path.  A predecessor that never calls
// grid_trigger lets it start when it ends, as an ordinary launch does.
BEM_D void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
BEM_D void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                                  A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

// -------------------------------------------------------------- complex ----
BEM_HD float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
BEM_HD double2 cmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
BEM_HD float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
BEM_HD double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
BEM_HD float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
BEM_HD double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
BEM_HD float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
BEM_HD double2 cscale(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

template <typename R> struct cplx;
template <> struct cplx<float> {
  typedef float2 type;
  static BEM_HD float2 make(float a, float b) { return make_float2(a, b); }
};
template <> struct cplx<double> {
  typedef double2 type;
  static BEM_HD double2 make(double a, double b) { return make_double2(a, b); }
};

// ------------------------------------------------------------ double-float --
struct df {
  float hi, lo;
};

BEM_D df two_sum(float a, float b) {
  float s = a + b;
  float bb = s - a;
  float e = (a - (s - bb)) + (b - bb);
  return {s, e};
}
BEM_D df quick_two_sum(float a, float b) {
  float s = a + b;
  return {s, b - (s - a)};
}
BEM_D df two_prod(float a, float b) {
  float p = a * b;
  return {p, fmaf(a, b, -p)};
}
BEM_D df df_add(df a, df b) {
  df s = two_sum(a.hi, b.hi);
  df t = two_sum(a.lo, b.lo);
  s.lo += t.hi;
  s = quick_two_sum(s.hi, s.lo);
  s.lo += t.lo;
  return quick_two_sum(s.hi, s.lo);
}
BEM_D df df_neg(df a) { return {-a.hi, -a.lo}; }
BEM_D df df_sub(df a, df b) { return df_add(a, df_neg(b)); }
BEM_D df df_mul(df a, df b) {
  df p = two_prod(a.hi, b.hi);
  p.lo = fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, p.lo));
  return quick_two_sum(p.hi, p.lo);
}
BEM_D df df_mul_f(df a, float b) {
  df p = two_prod(a.hi, b);
  p.lo = fmaf(a.lo, b, p.lo);
  return quick_two_sum(p.hi, p.lo);
}
// sqrt of a positive df: one Newton step on an FP32 root taken from the
// approximate reciprocal root.  The step removes the root's error to second
// order (relative error about 2^-44); a.hi <= 0 gives 0.
BEM_D float rsqrt_ftz(float x);
BEM_D df df_sqrt(df a) {
  if (!(a.hi > 0.0f)) return {0.0f, 0.0f};
  const float y = rsqrt_ftz(a.hi);
  const float s = a.hi * y;
  df s2 = two_prod(s, s);
  float r = ((a.hi - s2.hi) - s2.lo + a.lo) * (0.5f * y);
  return quick_two_sum(s, r);
}

// 2*pi as a three-term float expansion (hi + mid + lo), for argument reduction.
#define BEM_TWO_PI_HI 6.28318548202514648f
#define BEM_TWO_PI_MID -1.7484555314695172e-07f
#define BEM_TWO_PI_LO -6.8604980400235275e-15f
#define BEM_INV_TWO_PI 0.159154943091895336f
#define BEM_INV_FOUR_PI 0.0795774715459476678f

// Single-instruction approximations (PTX .approx.ftz: subnormal inputs and
// results flush to zero).  The library is built without -ftz, and the non-ftz
// forms of these PTX instructions carry subnormal handling around each one; the
// hot loops only apply them to arguments clamped well away from the subnormal
// range (r^2 >= 1e-30, |angle| <= pi + 1e-6).  Documented accuracy (PTX ISA):
// rsqrt/rcp about 2^-22 relative (rcp: 1 ulp), sin/cos 2^-20.5 absolute on [-pi, pi].
BEM_D float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
BEM_D float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
BEM_D void sincos_ftz(float x, float* s, float* c) {
  asm("sin.approx.ftz.f32 %0, %1;" : "=f"(*s) : "f"(x));
  asm("cos.approx.ftz.f32 %0, %1;" : "=f"(*c) : "f"(x));
}
// Nearest integer of |x| < 2^22 on the FMA pipe: adding 1.5 * 2^23 rounds away
// every fraction bit (round to nearest even); subtracting it back is exact.
// __fadd_rn / __fsub_rn are never contracted with a multiply that produced x, so
// the result is that of the rounded x in every inlined context.
BEM_D float round_nearest_small(float x) {
  const float kMagic = 12582912.0f;
  return __fsub_rn(__fadd_rn(x, kMagic), kMagic);
}

// sin x and cos x with RELATIVE accuracy for small |x| (sin(z/2) feeds
// 1 - cos z = 2 sin^2(z/2), where an absolute-accuracy approximation loses all
// relative accuracy as z -> 0).  x is reduced by the nearest multiple n*pi (pi
// split in two floats; each multiple flips both signs), then the Taylor series
// in x^2: sin to x^13, cos to x^12, coefficients (-1)^j / (2j+1)! and
// (-1)^j / (2j)!; the truncation error is below 7e-9 on |x| <= pi/2.
// For |x| < 2^20.
BEM_D void sincos_taylor(float x, float* s, float* c) {
  const float n = round_nearest_small(x * 0.318309873342514f);
  float r = fmaf(-n, 3.14159274101257324f, x);
  r = fmaf(-n, -8.742278012618954e-08f, r);
  const float r2 = r * r;
  float ps = 1.6059043836821613e-10f;
  ps = fmaf(ps, r2, -2.505210838544172e-08f);
  ps = fmaf(ps, r2, 2.7557319223985893e-06f);
  ps = fmaf(ps, r2, -1.984126984126984e-04f);
  ps = fmaf(ps, r2, 8.333333333333333e-03f);
  ps = fmaf(ps, r2, -1.6666666666666666e-01f);
  float sv = fmaf(ps * r2, r, r);
  float pc = 2.08767569878681e-09f;
  pc = fmaf(pc, r2, -2.755731922398589e-07f);
  pc = fmaf(pc, r2, 2.48015873015873e-05f);
  pc = fmaf(pc, r2, -1.388888888888889e-03f);
  pc = fmaf(pc, r2, 4.1666666666666664e-02f);
  pc = fmaf(pc, r2, -0.5f);
  float cv = fmaf(pc, r2, 1.0f);
  // (-1)^n from the parity of n (|n| < 2^20, exact in float)
  const bool odd = (((int)n) & 1) != 0;
  *s = odd ? -sv : sv;
  *c = odd ? -cv : cv;
}

// theta = a - 2*pi*rint(a / 2pi) for a df angle; the result lies in [-pi, pi]
// and is accurate to about 2^-44 * |a| + 2^-24.
BEM_D float df_reduce_two_pi(df a) {
  float n = rintf(a.hi * BEM_INV_TWO_PI);
  df t = two_prod(-n, BEM_TWO_PI_HI);  // exact -n*2pi_hi
  df r = df_add(a, t);
  r = df_add(r, two_prod(-n, BEM_TWO_PI_MID));
  return r.hi + (r.lo - n * BEM_TWO_PI_LO);
}

// Reduce an FP32 angle of moderate size (|t| < 2^20) into [-pi, pi].
BEM_D float reduce_two_pi(float t) {
  float n = round_nearest_small(t * BEM_INV_TWO_PI);
  t = fmaf(-n, BEM_TWO_PI_HI, t);
  return fmaf(-n, BEM_TWO_PI_MID, t);
}

// -------------------------------------------------------- FP64 on this part --
// FP64 issues at 1/64 of the FP32 rate here, so an FP64 kernel's time is its count of FP64
// instructions; everything else (table reads, FP32, integer work) is nearly free beside it.
//
// sin and cos of k r by table lookup and the addition theorem (P. T. P. Tang, Table-lookup
// algorithms for elementary functions and their error analysis, 1991), in units of
// h = 2 pi / 2048: u = r (k / h), n its nearest integer, x = u - n.  The table holds (cos, sin)
// of the first quadrant's 512 units; the other quadrants follow by exchanging and negating
// words, which is integer work.  With the units in the polynomials' coefficients there is no
// product k r and no reduction of it (k / h is held in two doubles, so x is exact to 2^-53 of
// a unit whatever u), and |x| <= 1/2 (pi / 2048) needs two Taylor terms each: sin to x^3 with
// the cubic coefficient moved by 0.87 of half a unit's x^5 / 120 (error 1e-17), cos to x^4
// (2e-20): 13 FP64 instructions for the pair, against 17 with 512 units to the circle, an
// angle in radians and its two-term reduction.
// Error: three roundings of 2^-54 (the table's entry, the two of the last combination) and the
// polynomial, 2e-16 absolute; for |k r| <= h / 2 the entry is (1, 0) and the sine's error is the
// polynomial's, below 1e-14 of it.  |u| < 2^31 (k r below 6.5e6).
constexpr int kSincosTable = 512, kSincosUnits = 4 * kSincosTable;
struct AngleUnits {
  double hi, lo;  // k / h
};
BEM_D AngleUnits angle_units(double k) {
  AngleUnits a;
  a.hi = k * 325.94932345220167;
  a.lo = fma(k, 325.94932345220167, -a.hi) + k * -2.0150964915386866e-14;
  return a;
}
// The table (kSincosTable entries) on the host: the first quadrant's (cos, sin) from the first
// octant by symmetry, in long double (an angle rounded to double moves an entry by as much as
// its own rounding does).  Formed once per process: 0.3 ms where long double is software.
inline const std::vector<double2>& sincos_table_host() {
  static const std::vector<double2> table = [] {
    std::vector<double2> t(kSincosTable);
    for (int i = 0; i < kSincosTable; ++i) {
      const int o = i < kSincosTable - i ? i : kSincosTable - i;
      const long double a = 2.0L * 3.14159265358979323846264338327950288L * o / kSincosUnits;
      const double c = (double)cosl(a), s = (double)sinl(a);
      t[i] = i == o ? make_double2(c, s) : make_double2(s, c);
    }
    return t;
  }();
  return table;
}
// The table into shared memory, by the whole CTA (synchronise before use): from its copy
// beside the mesh, or computed where there is none (src null; about 5% of a small CTA's FP64
// work).
BEM_D void load_sincos_table(double2* tab, const double2* src) {
  for (int i = threadIdx.x; i < kSincosTable; i += blockDim.x) {
    if (src != nullptr) {
      tab[i] = src[i];
    } else {
      double s, c;
      sincospi(i * (2.0 / kSincosUnits), &s, &c);
      tab[i] = make_double2(c, s);
    }
  }
}
BEM_D void sincos_table(double r, AngleUnits k, const double2* tab, double* s, double* c) {
  constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52: the sum's low word is the nearest integer
  const double t = fma(r, k.hi, kMagic);
  const double x = fma(r, k.lo, fma(r, k.hi, -(t - kMagic)));
  const int n = __double2loint(t);
  const double2 q = tab[n & (kSincosTable - 1)];
  // quadrant 0 (c, s), 1 (-s, c), 2 (-c, -s), 3 (s, -c)
  const bool odd = (n & kSincosTable) != 0;
  const int ssign = (n << 21) & 0x80000000, csign = ((n << 22) ^ (n << 21)) & 0x80000000;
  const double a = odd ? q.y : q.x, b = odd ? q.x : q.y;
  const double ec = __hiloint2double(__double2hiint(a) ^ csign, __double2loint(a));
  const double es = __hiloint2double(__double2hiint(b) ^ ssign, __double2loint(b));
  const double x2 = x * x;
  const double sx = x * fma(x2, -4.812807078551805e-09, 0.0030679615757712823);
  const double cm1 = x2 * fma(x2, 3.691377174997586e-12, -4.706194115204505e-06);  // cos - 1
  *c = fma(ec, cm1, fma(-es, sx, ec));
  *s = fma(es, cm1, fma(ec, sx, es));
}
// a == 0 for a sum of squares, in integer instructions.
BEM_D bool is_zero(double a) { return (__double2hiint(a) | __double2loint(a)) == 0; }

// Inverse of a pivot, 0 for d = 0.  Where |d|^2 or its reciprocal would leave the exponent
// range, d is multiplied by a power of two before and the result after, so a matrix scaled by
// one has the same multipliers to the bit.  pivot_inverse takes one reciprocal instead of two
// divisions (the register panels, where it is on the critical path of a step: LU of one
// matrix of order 520 takes 0.590 ms without a test of the range, 0.600 with the range known
// from the pivot's key, 0.603 tested on |d|^2, 0.613 with the scaling in line).
template <typename R> struct PivotRange;
template <> struct PivotRange<float> {
  static constexpr float lo = 0x1p-100f, hi = 0x1p100f, up = 0x1p80f, down = 0x1p-80f;
};
template <> struct PivotRange<double> {
  static constexpr double lo = 0x1p-900, hi = 0x1p900, up = 0x1p640, down = 0x1p-640;
};
BEM_D float rcp_round(float a) { return __frcp_rn(a); }
BEM_D double rcp_round(double a) { return __drcp_rn(a); }
template <bool DIV, typename C2> __device__ __noinline__ C2 pivot_inverse_scaled(C2 d) {
  using R = decltype(d.x);
  C2 r = d;
  if (d.x == R(0) && d.y == R(0)) return r;
  const R s = fma(d.x, d.x, d.y * d.y) < R(1) ? PivotRange<R>::up : PivotRange<R>::down;
  d.x *= s;
  d.y *= s;
  const R m = fma(d.x, d.x, d.y * d.y), rm = rcp_round(m);
  r.x = (DIV ? d.x / m : d.x * rm) * s;
  r.y = (DIV ? -d.y / m : -d.y * rm) * s;
  return r;
}
template <bool DIV, typename C2> BEM_D C2 pivot_inverse_plain(C2 d) {
  const auto m = fma(d.x, d.x, d.y * d.y);
  C2 r;
  if constexpr (DIV) {
    r.x = d.x / m;
    r.y = -d.y / m;
  } else {
    const auto rm = rcp_round(m);
    r.x = d.x * rm;
    r.y = -d.y * rm;
  }
  return r;
}
template <bool DIV = false, typename C2> BEM_D C2 pivot_inverse(C2 d) {
  using R = decltype(d.x);
  const R m = fma(d.x, d.x, d.y * d.y);
  return m >= PivotRange<R>::lo && m <= PivotRange<R>::hi ? pivot_inverse_plain<DIV>(d) : pivot_inverse_scaled<DIV>(d);
}

// ------------------------------------------------------- row permutation --
// Applies a panel's net row permutation (cnt <= 128 pairs: row sdst takes row ssrc) to one
// column of n entries, by one warp: every source row is loaded (at most 4 per lane, all in
// flight) before any destination row is stored.
template <typename T>
__device__ __forceinline__ void permute_column(T* a, int n, int cnt, const int* sdst, const int* ssrc) {
  const int lane = threadIdx.x & 31;
  T v[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = lane + 32 * q;
    if (e < cnt && (unsigned)ssrc[e] < (unsigned)n) v[q] = a[ssrc[e]];
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int e = lane + 32 * q;
    if (e < cnt && (unsigned)ssrc[e] < (unsigned)n && (unsigned)sdst[e] < (unsigned)n) a[sdst[e]] = v[q];
  }
}

// -------------------------------------------------------- status / limits --
// Device status word written by kernels that can detect bad input; the host
// reads it after the launch.  No kernel traps or spins without a bound.
enum BemDeviceStatus : int {
  BEM_DEV_OK = 0,
  BEM_DEV_ZERO_PIVOT = 1,
  BEM_DEV_NONFINITE = 2,
};
