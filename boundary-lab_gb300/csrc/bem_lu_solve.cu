// Solves and refinement of the mixed form's FP32 LU factors (sm_103a).
//
// A triangular solve of one right-hand side reads each factor entry once, so its floor is
// the HBM time of one matrix; what it took before was the latency of one 32-row
// substitution, one cluster barrier and one strip update after another (n = 4,976: 312
// steps of 6 us, 1.88 ms a solve whether 1 or 15 matrices were in flight).  Here the
// 256 x 256 diagonal blocks of both factors are inverted once per factorisation, all of
// them side by side (lu_block_inverse_kernel), so a solve has two cluster barriers per 256
// rows and no serial chain inside a block: x_K = inv(L_KK) b_K is a matrix-vector product
// shared by the cluster's CTAs, and so is the update of the rows below.  One solve: 1.88 ->
// 0.43 ms for one matrix of order 4,976, 0.68 ms for 15 (0.44 ms is their HBM time); 153 ->
// 33 us at order 518; the inverses take 0.09 ms (one), 0.34 ms (16 of
// order 2,524).
//
// The substitution arithmetic stays FP32; the refinement loop around it takes the residual
// of the FP32 matrix with exact products and compensated sums as before.
//
// Every spin is a hardware cluster barrier; every CTA of a cluster runs the same sequence.
#include <cooperative_groups.h>

#include <type_traits>

#include "bem_common.cuh"
#include "bem_kernels.h"

namespace cg = cooperative_groups;

namespace bem {
namespace {

constexpr int kInvWarps = 8, kInvStages = 4;
constexpr int kInvBlk = kOuterBlock / 32;

template <int CPW> constexpr size_t inverse_smem() {
  return ((size_t)kInvStages * 32 * 32 + (size_t)kInvWarps * kOuterBlock * CPW) * sizeof(float2);
}

// inv[(mat, block K, side)] = inverse of the unit lower (side 0) or the upper (side 1)
// triangle of diagonal block K, column-major 256 x 256; rows and columns beyond the matrix
// are zero.  The upper triangle is taken in reversed row and column order, where it is a
// lower one, so both sides run the same left-looking substitution: a warp owns CPW columns
// of the identity, lane = row of the current 32-row block, the 32 x 32 tiles of the triangle
// pass through shared memory once per CTA (the scheme of lu_urows_kernel).  A slab (the
// CTA's 8 CPW columns) starts at the block row of its columns: the rows above are zero.
// Grid (256 / (8 CPW) slabs x 2 sides, blocks, batch).  Bound by latency (the substitutions'
// shuffles) at two warps per scheduler, so eight warps of four columns share a tile where
// four of eight did: 32 matrices of order 600 348 -> 225 us, one of order 520 48 -> 35.
template <int SIDE, int CPW>
__device__ void block_inverse(const float2* __restrict__ D, long long lda, int KB, float2* __restrict__ out, int col0,
                              float2* ring, float2* X) {
  const int slab = col0 >> 5;  // first block row
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  constexpr bool REV = SIDE == 1;
  int pb = slab, pl = slab;
  auto stage = [&](int slot) {
    if (pb < kInvBlk) {
      float2* dst = ring + (size_t)slot * 32 * 32;
      const int rb = REV ? kInvBlk - 1 - pb : pb, cb = REV ? kInvBlk - 1 - pl : pl;
#pragma unroll
      for (int q = 0; q < 16 / kInvWarps; ++q) {
        const int i = threadIdx.x + 32 * kInvWarps * q, col = i >> 4, piece = i & 15;
        const int c = 32 * cb + col, r = 32 * rb + 2 * piece;
        // entries beyond the matrix are zero-filled (a piece may straddle its last row)
        const int bytes = c < KB ? min(max(KB - r, 0), 2) * (int)sizeof(float2) : 0;
        const float2* src = bytes > 0 ? D + (size_t)c * lda + r : D;
        const unsigned d = (unsigned)__cvta_generic_to_shared(dst + 32 * col + 2 * piece);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes));
      }
      if (++pl > pb) {
        pl = slab;
        ++pb;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = 0; i < kInvStages - 1; ++i) stage(i);
  const int c0 = col0 + wid * CPW;  // this warp's first column, in the side's order
  float2 x[CPW];
  int t = 0;
  for (int b = slab; b < kInvBlk; ++b) {
#pragma unroll
    for (int c = 0; c < CPW; ++c) x[c] = make_float2(32 * b + lane == c0 + c ? 1.f : 0.f, 0.f);
    for (int l = slab; l <= b; ++l, ++t) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kInvStages - 2) : "memory");
      __syncthreads();  // tile t is in place for every warp, and tile t - 1 is no longer read
      stage((t + kInvStages - 1) % kInvStages);
      const float2* T = ring + (size_t)(t % kInvStages) * 32 * 32;
      const int rl = REV ? 31 - lane : lane;
      if (l < b) {
        const float4* xs = reinterpret_cast<const float4*>(X + (size_t)32 * l * CPW);
#pragma unroll 8
        for (int kk = 0; kk < 32; ++kk) {
          const float2 lv = T[32 * (REV ? 31 - kk : kk) + rl];
#pragma unroll
          for (int q = 0; q < CPW / 2; ++q) {
            const float4 u = xs[kk * (CPW / 2) + q];
            x[2 * q].x = fmaf(-lv.x, u.x, fmaf(lv.y, u.y, x[2 * q].x));
            x[2 * q].y = fmaf(-lv.x, u.y, fmaf(-lv.y, u.x, x[2 * q].y));
            x[2 * q + 1].x = fmaf(-lv.x, u.z, fmaf(lv.y, u.w, x[2 * q + 1].x));
            x[2 * q + 1].y = fmaf(-lv.x, u.w, fmaf(-lv.y, u.z, x[2 * q + 1].y));
          }
        }
        continue;
      }
      float2 dinv = make_float2(1.f, 0.f);
      if (REV) dinv = pivot_inverse<true>(T[32 * rl + rl]);  // zero beyond the matrix
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float2 lv = T[32 * (REV ? 31 - j : j) + rl];
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
          if (REV && lane == j) x[c] = cmul(x[c], dinv);
          const float xr = __shfl_sync(0xffffffffu, x[c].x, j), xi = __shfl_sync(0xffffffffu, x[c].y, j);
          if (lane > j) {
            x[c].x = fmaf(-lv.x, xr, fmaf(lv.y, xi, x[c].x));
            x[c].y = fmaf(-lv.x, xi, fmaf(-lv.y, xr, x[c].y));
          }
        }
      }
    }
    float4* xd = reinterpret_cast<float4*>(X + (size_t)(32 * b + lane) * CPW);
#pragma unroll
    for (int q = 0; q < CPW / 2; ++q) xd[q] = make_float4(x[2 * q].x, x[2 * q].y, x[2 * q + 1].x, x[2 * q + 1].y);
    __syncwarp();
    const int row = 32 * b + lane;
#pragma unroll
    for (int c = 0; c < CPW; ++c) {
      const int r = REV ? kOuterBlock - 1 - row : row, cc = REV ? kOuterBlock - 1 - (c0 + c) : c0 + c;
      const bool in = r < KB && cc < KB;
      out[(size_t)cc * kOuterBlock + r] = in ? x[c] : make_float2(0.f, 0.f);
    }
  }
}

template <int CPW>
__global__ void __launch_bounds__(kInvWarps * 32) lu_block_inverse_kernel(const float2* __restrict__ A, long long lda,
                                                                          long long strideA, int n,
                                                                          float2* __restrict__ inv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* ring = reinterpret_cast<float2*>(smem_raw);  // [stage][column][row]
  float2* X = ring + kInvStages * 32 * 32 + (size_t)(threadIdx.x >> 5) * kOuterBlock * CPW;  // [row][column]
  const int col0 = (blockIdx.x >> 1) * kInvWarps * CPW, side = blockIdx.x & 1, K = blockIdx.y;
  const int KB = min(kOuterBlock, n - K * kOuterBlock);
  const float2* D = A + (size_t)blockIdx.z * strideA + (size_t)K * kOuterBlock * (lda + 1);
  float2* out = inv + (((size_t)blockIdx.z * gridDim.y + K) * 2 + side) * kOuterBlock * kOuterBlock;
  if (side == 0)
    block_inverse<0, CPW>(D, lda, KB, out, col0, ring, X);
  else
    block_inverse<1, CPW>(D, lda, KB, out, col0, ring, X);
}

// ------------------------------------------------------------------ solves --
// One cluster per (matrix, group of NR right-hand sides).  Rows are dealt to the CTAs in
// blocks of 32 (block rb to CTA rb mod CL), so every outer block and every trailing part is
// spread evenly.  Per outer block K, forward then backward:
//  1. the owners of K's row blocks push their current right-hand sides into every CTA;
//     cluster barrier;
//  2. each owner multiplies its 32 rows of the block's inverse by them (16 warps share the
//     columns, partial sums added in a fixed order) and pushes its x into every CTA; barrier;
//  3. every CTA subtracts the block's columns times x from its rows below (above): a task is
//     a row block and a quarter of the 256 columns, lanes along the rows, so every load of a
//     warp is one run of 256 bytes with kLoads of them in flight; each quarter has a partial
//     sum of its own per row, so no two warps add to the same place.
constexpr int kSolveThreads = 512, kSolveWarps = kSolveThreads / 32, kQuarters = 4;

size_t solve_smem(int n, int cl, int nr) {
  const int nrb = (n + 31) / 32, nloc = (nrb + cl - 1) / cl;
  return ((size_t)nloc * 32 * (1 + kQuarters) + 2 * kOuterBlock + kSolveWarps * 32) * nr * sizeof(float2);
}

template <int NR>
__global__ void __launch_bounds__(kSolveThreads, 1) lu_solve_blocks_kernel(const float2* __restrict__ A, long long lda,
                                                                        long long strideA, int n,
                                                                        const float2* __restrict__ inv,
                                                                        const int* __restrict__ perm, float2* B,
                                                                        long long ldb, int groups) {
  constexpr int kLoads = NR == 1 ? 32 : 16;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), CL = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int mat = blockIdx.y / groups, group = blockIdx.y - mat * groups;
  const int nrb = (n + 31) / 32, nloc = (nrb + CL - 1) / CL, nouter = (n + kOuterBlock - 1) / kOuterBlock;
  const float2* M = A + (size_t)mat * strideA;
  const float2* Inv = inv + (size_t)mat * nouter * 2 * kOuterBlock * kOuterBlock;
  float2* b = B + ((size_t)mat * groups + group) * NR * ldb;
  const int* pm = perm + (size_t)mat * n;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* xs = reinterpret_cast<float2*>(smem_raw);        // [NR][nloc x 32]: my rows
  float2* part = xs + (size_t)NR * nloc * 32;              // [quarter][NR][nloc x 32]
  float2* pb = part + (size_t)kQuarters * NR * nloc * 32;  // [NR][256]: the block's right-hand sides
  float2* yv = pb + NR * kOuterBlock;                      // [NR][256]: the block's x
  float2* red = yv + NR * kOuterBlock;                     // [warp][NR][32]
  const int loc = nloc * 32;
  for (int i = tid; i < loc; i += kSolveThreads) {
    const int r = ((i >> 5) * CL + rank) * 32 + lane;
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      xs[c * loc + i] = r < n ? b[c * ldb + pm[r]] : make_float2(0.f, 0.f);
#pragma unroll
      for (int q = 0; q < kQuarters; ++q) part[(q * NR + c) * loc + i] = make_float2(0.f, 0.f);
    }
  }
  cluster.sync();  // every CTA has read b before anyone writes it back
  for (int step = 0; step < 2 * nouter; ++step) {
    const bool fwd = step < nouter;
    const int K = fwd ? step : 2 * nouter - 1 - step;
    const int rb0 = K * kInvBlk, nb = min(kInvBlk, nrb - rb0);  // the block's row blocks
    const float2* V = Inv + ((size_t)K * 2 + (fwd ? 0 : 1)) * kOuterBlock * kOuterBlock;
    // 1. current right-hand sides of my row blocks, to every CTA (a warp per target and row block)
    for (int w = wid; w < nb * CL; w += kSolveWarps) {
      const int lb = w / CL, target = w - lb * CL;
      if ((rb0 + lb) % CL != rank) continue;
      const int i = ((rb0 + lb) / CL) * 32 + lane;
#pragma unroll
      for (int c = 0; c < NR; ++c) {
        float2 v = xs[c * loc + i];
#pragma unroll
        for (int q = 0; q < kQuarters; ++q) v = csub(v, part[(q * NR + c) * loc + i]);
        *cluster.map_shared_rank(&pb[c * kOuterBlock + 32 * lb + lane], target) = v;
      }
    }
    cluster.sync();
    // 2. my rows of x
    for (int lb = 0; lb < nb; ++lb) {
      if ((rb0 + lb) % CL != rank) continue;
      // columns of the triangle's inverse that reach this row block, shared out over the warps
      const int j0 = fwd ? 0 : 32 * lb, per = fwd ? 2 * (lb + 1) : 2 * (nb - lb);
      float2 acc[NR];
#pragma unroll
      for (int c = 0; c < NR; ++c) acc[c] = make_float2(0.f, 0.f);
      const float2* col = V + (size_t)(j0 + wid * per) * kOuterBlock + 32 * lb + lane;
      const float2* xb = pb + j0 + wid * per;
      float2 v[16];  // per <= 16: all loads in flight at once
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = j < per ? col[(size_t)j * kOuterBlock] : make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (j >= per) break;
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          const float2 u = xb[c * kOuterBlock + j];
          acc[c].x = fmaf(v[j].x, u.x, fmaf(-v[j].y, u.y, acc[c].x));
          acc[c].y = fmaf(v[j].x, u.y, fmaf(v[j].y, u.x, acc[c].y));
        }
      }
#pragma unroll
      for (int c = 0; c < NR; ++c) red[(wid * NR + c) * 32 + lane] = acc[c];
      __syncthreads();
      // a warp per target sums the partials again rather than wait for one more barrier
      for (int target = wid; target < CL; target += kSolveWarps) {
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          float2 v = make_float2(0.f, 0.f);
#pragma unroll
          for (int w = 0; w < kSolveWarps; ++w) v = cadd(v, red[(w * NR + c) * 32 + lane]);
          *cluster.map_shared_rank(&yv[c * kOuterBlock + 32 * lb + lane], target) = v;
          if (target == rank) {  // x of the forward pass is the right-hand side of the backward one
            const int i = ((rb0 + lb) / CL) * 32 + lane;
            xs[c * loc + i] = v;
#pragma unroll
            for (int q = 0; q < kQuarters; ++q) part[(q * NR + c) * loc + i] = make_float2(0.f, 0.f);
          }
        }
      }
      __syncthreads();  // red is free for the next row block
    }
    cluster.sync();
    // 3. my rows of the other blocks
    const int first = fwd ? rb0 + nb : 0, last = fwd ? nrb : rb0;  // row blocks [first, last)
    const int l0 = first <= rank ? 0 : (first - rank + CL - 1) / CL, l1 = last <= rank ? 0 : (last - rank + CL - 1) / CL;
    const int kcols = min(kOuterBlock, n - K * kOuterBlock);
    for (int task = wid; task < (l1 - l0) * kQuarters; task += kSolveWarps) {
      const int li = l0 + (task >> 2), q = task & 3;
      const int r = (li * CL + rank) * 32 + lane;
      const int jn = min(64, kcols - 64 * q);
      float2 acc[NR];
#pragma unroll
      for (int c = 0; c < NR; ++c) acc[c] = part[(q * NR + c) * loc + li * 32 + lane];
      const float2* col = M + (size_t)(K * kOuterBlock + 64 * q) * lda + min(r, n - 1);
      const float2* y = yv + 64 * q;
      int j = 0;
      for (; j + kLoads <= jn; j += kLoads) {
        float2 v[kLoads];
#pragma unroll
        for (int u = 0; u < kLoads; ++u) v[u] = col[(size_t)(j + u) * lda];
#pragma unroll
        for (int u = 0; u < kLoads; ++u)
#pragma unroll
          for (int c = 0; c < NR; ++c) {
            const float2 w = y[c * kOuterBlock + j + u];
            acc[c].x = fmaf(v[u].x, w.x, fmaf(-v[u].y, w.y, acc[c].x));
            acc[c].y = fmaf(v[u].x, w.y, fmaf(v[u].y, w.x, acc[c].y));
          }
      }
      for (; j < jn; ++j) {
        const float2 v = col[(size_t)j * lda];
#pragma unroll
        for (int c = 0; c < NR; ++c) {
          const float2 w = y[c * kOuterBlock + j];
          acc[c].x = fmaf(v.x, w.x, fmaf(-v.y, w.y, acc[c].x));
          acc[c].y = fmaf(v.x, w.y, fmaf(v.y, w.x, acc[c].y));
        }
      }
#pragma unroll
      for (int c = 0; c < NR; ++c) part[(q * NR + c) * loc + li * 32 + lane] = acc[c];
    }
    __syncthreads();
  }
  for (int i = tid; i < loc; i += kSolveThreads) {
    const int r = ((i >> 5) * CL + rank) * 32 + lane;
    if (r < n)
#pragma unroll
      for (int c = 0; c < NR; ++c) b[c * ldb + r] = xs[c * loc + i];
  }
  cluster.sync();  // no CTA leaves while others may still write its shared memory
}

// -------------------------------------------------------------- refinement --
// x (+)= d, and x as float hi / lo pairs (re hi, im hi, re lo, im lo) for the residual, so
// that it runs no FP64 instruction in its inner loop.  A system (blockIdx.y) whose residual is
// within tol stays as it is while others of its batch are refined, so that its x does not
// depend on them; the test is the host's, to the bit.
template <bool FIRST>
__global__ void update_x_kernel(const double* __restrict__ norms, double tol, const float2* __restrict__ d,
                                double2* __restrict__ x, float4* __restrict__ xs, long long ldb) {
  if (blockIdx.x * blockDim.x + threadIdx.x >= ldb) return;
  const long long i = blockIdx.y * ldb + blockIdx.x * blockDim.x + threadIdx.x;
  if (!FIRST) {
    const double r2 = norms[2 * blockIdx.y], b2 = norms[2 * blockIdx.y + 1];
    if ((b2 > 0.0 ? sqrt(r2 / b2) : sqrt(r2)) <= tol) return;
  }
  const float2 dv = d[i];
  double2 v = make_double2((double)dv.x, (double)dv.y);
  if (!FIRST) {
    const double2 o = x[i];
    v.x += o.x;
    v.y += o.y;
  }
  x[i] = v;
  const float hr = (float)v.x, hi = (float)v.y;
  xs[i] = make_float4(hr, hi, (float)(v.x - (double)hr), (float)(v.y - (double)hi));
}

// One exact product into a compensated sum: p = a xh is added to (sh, sl) by two_sum, and
// its rounding error and a xl to e in FP32, so the sum carries about 2^-40 relative error
// per 256 columns, far below the 1e-10 refinement target.
__device__ __forceinline__ void acc_exact_prod(float& sh, float& sl, float& e, float a, float xh, float xl) {
  const float p = a * xh;
  const float pe = fmaf(a, xh, -p);
  const float t = sh + p;
  const float bb = t - sh;
  sl += (sh - (t - bb)) + (p - bb);
  sh = t;
  e = fmaf(a, xl, e + pe);
}

// part[split] = A x over the split's columns, with A in FP32 and x in FP64: every product
// a * (x_hi + x_lo) is formed exactly (two FMAs) and summed in double-float, so the sums
// carry the accuracy of an FP64 product with the FP32 matrix at the FP32 rate (FP64 issues
// at 1/64 of it here).  A CTA covers 64 rows; its four groups of 64 threads take
// interleaved 64-column slices of each 256-column block of x staged in shared memory, each
// thread keeping two independent double-float sums (even / odd columns).  gridDim.y splits
// of the columns fill the GPU when few systems are in flight (one matrix of order 4,976:
// 78 CTAs and 0.54 ms unsplit, 0.08 ms with eight splits).
__global__ void __launch_bounds__(256) residual_parts_kernel(const float2* __restrict__ A, long long lda,
                                                             long long strideA, int n, const float4* __restrict__ xs,
                                                             long long ldb, int nrhs, int cols_per_split,
                                                             double2* __restrict__ part) {
  __shared__ float4 xsh[256];
  __shared__ double sum[2][4][64];
  const int rl = threadIdx.x & 63, cgp = threadIdx.x >> 6;
  const int row = blockIdx.x * 64 + rl;
  const int sys = blockIdx.z, mat = sys / nrhs;
  const int c_lo = blockIdx.y * cols_per_split, c_hi = min(n, c_lo + cols_per_split);
  const float2* M = A + (size_t)mat * strideA;
  const float4* xv = xs + (size_t)sys * ldb;
  float srh = 0.f, srl = 0.f, er = 0.f, sih = 0.f, sil = 0.f, ei = 0.f;      // even columns
  float trh = 0.f, trl = 0.f, fr = 0.f, tih = 0.f, til = 0.f, fi = 0.f;      // odd columns
  for (int j0 = c_lo; j0 < c_hi; j0 += 256) {
    __syncthreads();
    {
      const int j = j0 + threadIdx.x;
      xsh[threadIdx.x] = j < c_hi ? xv[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const int cb = j0 + cgp * 64;
    const int jn = min(64, c_hi - cb);
    if (row < n && jn > 0) {
      const float2* col = M + (size_t)cb * lda + row;
      const float4* xg = xsh + cgp * 64;
      // sixteen columns' loads in flight, then their products (a loop of single columns waited
      // for memory at each: 58 us for 512 columns); columns beyond the split are zeros
#pragma unroll 1
      for (int t = 0; t < jn; t += 16) {
        float2 a[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) a[u] = t + u < jn ? col[(size_t)(t + u) * lda] : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 16; u += 2) {
          const float4 x0 = xg[t + u], x1 = xg[t + u + 1];
          // re += a.x xr - a.y xi ; im += a.x xi + a.y xr
          acc_exact_prod(srh, srl, er, a[u].x, x0.x, x0.z);
          acc_exact_prod(srh, srl, er, -a[u].y, x0.y, x0.w);
          acc_exact_prod(sih, sil, ei, a[u].x, x0.y, x0.w);
          acc_exact_prod(sih, sil, ei, a[u].y, x0.x, x0.z);
          acc_exact_prod(trh, trl, fr, a[u + 1].x, x1.x, x1.z);
          acc_exact_prod(trh, trl, fr, -a[u + 1].y, x1.y, x1.w);
          acc_exact_prod(tih, til, fi, a[u + 1].x, x1.y, x1.w);
          acc_exact_prod(tih, til, fi, a[u + 1].y, x1.x, x1.z);
        }
      }
    }
  }
  sum[0][cgp][rl] = ((double)srh + ((double)srl + (double)er)) + ((double)trh + ((double)trl + (double)fr));
  sum[1][cgp][rl] = ((double)sih + ((double)sil + (double)ei)) + ((double)tih + ((double)til + (double)fi));
  __syncthreads();
  if (cgp == 0 && row < n) {
    double2* p = part + ((size_t)blockIdx.y * gridDim.z + sys) * ldb;
    p[row] = make_double2(((sum[0][0][rl] + sum[0][1][rl]) + sum[0][2][rl]) + sum[0][3][rl],
                          ((sum[1][0][rl] + sum[1][1][rl]) + sum[1][2][rl]) + sum[1][3][rl]);
  }
}

// r = b - (sum of the splits' parts), rounded to FP32 into d for the next solve, with
// out[2 sys] = ||r||^2 and out[2 sys + 1] = ||b||^2 (b is FP32: the right-hand side as
// assembled).  One CTA per system, sums in a fixed order.
__global__ void __launch_bounds__(512) residual_finish_kernel(const double2* __restrict__ part, int splits,
                                                              const float2* __restrict__ b, long long ldb, int n,
                                                              float2* __restrict__ d, double* __restrict__ out) {
  const int sys = blockIdx.x, systems = gridDim.x;
  const float2* bv = b + (size_t)sys * ldb;
  float2* dv = d + (size_t)sys * ldb;
  double sr = 0.0, sb = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    double2 ax = part[(size_t)sys * ldb + i];
    for (int s = 1; s < splits; ++s) {
      const double2 p = part[((size_t)s * systems + sys) * ldb + i];
      ax.x += p.x;
      ax.y += p.y;
    }
    const float2 bb = bv[i];
    const double rx = (double)bb.x - ax.x, ry = (double)bb.y - ax.y;
    dv[i] = make_float2((float)rx, (float)ry);
    sr += rx * rx + ry * ry;
    sb += (double)bb.x * (double)bb.x + (double)bb.y * (double)bb.y;
  }
  __shared__ double s1[16], s2[16];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sr += __shfl_xor_sync(0xffffffffu, sr, o);
    sb += __shfl_xor_sync(0xffffffffu, sb, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s1[threadIdx.x >> 5] = sr;
    s2[threadIdx.x >> 5] = sb;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0, c = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      a += s1[w];
      c += s2[w];
    }
    out[2 * sys] = a;
    out[2 * sys + 1] = c;
  }
}

constexpr int kSolveCluster = 8;
constexpr size_t kSolveSmemMax = 220 * 1024;

}  // namespace

// Column splits of the residual: enough CTAs for four per SM.
int residual_splits(int n, int systems) {
  const long long ctas = (long long)((n + 63) / 64) * systems;
  int s = 1;
  while (s < kResidualSplits && ctas * s < 4LL * sm_count() && n >= 512 * s) s *= 2;
  return s;
}

size_t lu_inverse_bytes(int n, int batch) {
  return (size_t)batch * ((n + kOuterBlock - 1) / kOuterBlock) * 2 * kOuterBlock * kOuterBlock * sizeof(float2);
}

// Orders whose rows fit the cluster's shared memory (up to 43,264, with one right-hand side at a
// time); a larger one keeps the substitution of lu_solve_cluster_batched.
bool lu_solve_blocks_fits(int n) { return solve_smem(n, kSolveCluster, 1) <= kSolveSmemMax; }

cudaError_t lu_block_inverses(const void* LU, long long lda, int n, int batch, void* inv, cudaStream_t stream) {
  const int blocks = (n + kOuterBlock - 1) / kOuterBlock;
  auto run = [&](auto cpw_c) {
    constexpr int CPW = decltype(cpw_c)::value;
    constexpr size_t sm = inverse_smem<CPW>();
    ensure_smem_limit((const void*)lu_block_inverse_kernel<CPW>, sm);
    dim3 g(2 * kOuterBlock / (kInvWarps * CPW), blocks, batch);
    lu_block_inverse_kernel<CPW><<<g, kInvWarps * 32, sm, stream>>>((const float2*)LU, lda, lda * (long long)n, n,
                                                                    (float2*)inv);
    return cudaGetLastError();
  };
  // 4 columns per warp need fewer shared-memory reads per FMA; 2 shorten the chain of a
  // call that leaves SMs idle
  if (2LL * 8 * blocks * batch >= 2LL * sm_count()) return run(std::integral_constant<int, 4>{});
  return run(std::integral_constant<int, 2>{});
}

cudaError_t lu_solve_blocks_batched(const void* LU, long long lda, int n, int batch, const void* inv, const int* perm,
                                    void* B, long long ldb, int nrhs, cudaStream_t stream) {
  // right-hand sides of one matrix share its reads as far as their rows fit in shared memory
  int nr = nrhs;
  while (nr > 1 && (nrhs % nr != 0 || solve_smem(n, kSolveCluster, nr) > kSolveSmemMax)) --nr;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kSolveCluster, (unsigned)(batch * (nrhs / nr)));
  cfg.blockDim = dim3(kSolveThreads);
  cfg.dynamicSmemBytes = solve_smem(n, kSolveCluster, nr);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kSolveCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  auto run = [&](auto kern) {
    ensure_smem_limit((const void*)kern, cfg.dynamicSmemBytes);
    return cudaLaunchKernelEx(&cfg, kern, (const float2*)LU, lda, lda * (long long)n, n, (const float2*)inv, perm,
                              (float2*)B, ldb, nrhs / nr);
  };
  switch (nr) {
    case 1: return run(lu_solve_blocks_kernel<1>);
    case 2: return run(lu_solve_blocks_kernel<2>);
    case 3: return run(lu_solve_blocks_kernel<3>);
    default: return run(lu_solve_blocks_kernel<4>);
  }
}

cudaError_t refine_update_x(const double* norms, double tol, const float2* d, double2* x, void* xsplit, long long ldb,
                            int systems, cudaStream_t stream) {
  const dim3 grid((unsigned)((ldb + 255) / 256), systems);
  if (norms == nullptr)
    update_x_kernel<true><<<grid, 256, 0, stream>>>(norms, tol, d, x, (float4*)xsplit, ldb);
  else
    update_x_kernel<false><<<grid, 256, 0, stream>>>(norms, tol, d, x, (float4*)xsplit, ldb);
  return cudaGetLastError();
}

cudaError_t refine_residual(const void* A, long long lda, int n, int batch, const void* xsplit, const float2* b,
                            long long ldb, int nrhs, double2* parts, float2* d, double* norms, cudaStream_t stream,
                            int rule_batch) {
  const int systems = batch * nrhs, splits = residual_splits(n, (rule_batch > 0 ? rule_batch : batch) * nrhs);
  const int cols = ((n + splits - 1) / splits + 63) / 64 * 64;
  const int used = (n + cols - 1) / cols;
  dim3 g((n + 63) / 64, used, systems);
  residual_parts_kernel<<<g, 256, 0, stream>>>((const float2*)A, lda, lda * (long long)n, n, (const float4*)xsplit, ldb,
                                               nrhs, cols, parts);
  residual_finish_kernel<<<systems, 512, 0, stream>>>(parts, used, b, ldb, n, d, norms);
  return cudaGetLastError();
}

}  // namespace bem
