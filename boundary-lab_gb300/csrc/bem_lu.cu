// Dense complex LU with partial pivoting: driver, trailing updates and U rows (sm_103a).
//
// The reference solves each Burton-Miller system with CUDA.jl's `\`
// (cuSOLVER getrf + getrs, src/blab/solvers/julia_local/src/
// BeatEngineCore.jl:1206) and refactors for every channel.  Here the matrix of
// one frequency is factored once and every excitation is solved against the
// factors; many frequencies are factored together as a batch so that
// panel-factorisation latency of one matrix overlaps the work of others.
//
// Blocked right-looking LU, per block column k of width nb:
//   lu_panel_kernel   pivot search (|re|+|im| as LAPACK's icamax), row swap,
//                     scaling and rank-1 updates inside the panel; one CTA per
//                     matrix of the batch
//   lu_swap_kernel    the panel's row interchanges applied to the other columns
//   lu_trsm_kernel    U12 = L11^{-1} A12 (unit lower), L11 staged in shared memory
//   trailing update   A22 -= L21 U12 : a batched complex GEMM
#include <cublas_v2.h>

#include <vector>

#include "bem_common.cuh"
#include "bem_kernels.h"

namespace bem {
namespace {

template <typename R> struct CT;
template <> struct CT<float> { typedef float2 C2; };
template <> struct CT<double> { typedef double2 C2; };

template <typename C2> __device__ __forceinline__ auto cabs1(C2 v) -> decltype(v.x) { return fabs(v.x) + fabs(v.y); }

template <typename R>
__global__ void __launch_bounds__(1024) lu_panel_kernel(typename CT<R>::C2* A, long long lda, long long strideA, int n,
                                                        int k, int kb, int* ipiv, int* info) {
  typedef typename CT<R>::C2 C2;
  C2* M = A + (size_t)blockIdx.x * strideA;
  int* piv = ipiv + (size_t)blockIdx.x * n;
  __shared__ R s_val[32];
  __shared__ int s_idx[32];
  __shared__ C2 s_row[64];
  __shared__ int s_p;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
  for (int j = 0; j < kb; ++j) {
    const int col = k + j;
    const C2* Mc = M + (size_t)col * lda;
    R best = R(-1);
    int bi = n;
    for (int r = col + tid; r < n; r += blockDim.x) {
      R v = cabs1(Mc[r]);
      if (v > best) {  // first maximum in row order within this thread's stride
        best = v;
        bi = r;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      R ov = __shfl_xor_sync(0xffffffffu, best, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if (lane == 0) {
      s_val[wid] = best;
      s_idx[wid] = bi;
    }
    __syncthreads();
    if (wid == 0) {
      best = lane < nw ? s_val[lane] : R(-1);
      bi = lane < nw ? s_idx[lane] : n;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        R ov = __shfl_xor_sync(0xffffffffu, best, o);
        int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) {
          best = ov;
          bi = oi;
        }
      }
      if (lane == 0) {
        s_p = bi < n ? bi : col;
        piv[col] = s_p;
      }
    }
    __syncthreads();
    const int p = s_p;
    if (p != col) {
      for (int c = tid; c < kb; c += blockDim.x) {
        C2* a = M + (size_t)(k + c) * lda;
        C2 t = a[col];
        a[col] = a[p];
        a[p] = t;
      }
    }
    __syncthreads();
    for (int c = tid; c < kb; c += blockDim.x) s_row[c] = M[(size_t)(k + c) * lda + col];
    __syncthreads();
    const C2 d = s_row[j];
    C2 inv;
    if (d.x == R(0) && d.y == R(0)) {
      inv.x = R(0);
      inv.y = R(0);
      if (tid == 0 && info[blockIdx.x] == 0) info[blockIdx.x] = col + 1;
    } else {
      inv = pivot_inverse<true>(d);
    }
    for (int r = col + 1 + tid; r < n; r += blockDim.x) {
      C2 l = cmul(M[(size_t)col * lda + r], inv);
      M[(size_t)col * lda + r] = l;
      for (int c = j + 1; c < kb; ++c) {
        C2* a = M + (size_t)(k + c) * lda + r;
        C2 u = s_row[c];
        C2 v = *a;
        v.x -= l.x * u.x - l.y * u.y;
        v.y -= l.x * u.y + l.y * u.x;
        *a = v;
      }
    }
    __syncthreads();
  }
}

template <typename C2>
__global__ void lu_swap_kernel(C2* A, long long lda, long long strideA, int n, int k, int kb, const int* ipiv) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int ncols = n - kb;
  if (t >= ncols) return;
  const int c = t < k ? t : t + kb;
  C2* a = A + (size_t)blockIdx.y * strideA + (size_t)c * lda;
  const int* piv = ipiv + (size_t)blockIdx.y * n;
  for (int j = 0; j < kb; ++j) {
    const int r1 = k + j, r2 = piv[k + j];
    if (r2 != r1) {
      C2 tmp = a[r1];
      a[r1] = a[r2];
      a[r2] = tmp;
    }
  }
}

// U12 = L11^{-1} A12 for rows [k, k+kb) and columns [c_begin, c_end), with L11 the
// unit lower triangle of A[k:k+kb, k:k+kb]; blockDim columns per CTA.  The
// column block is staged through shared memory with coalesced loads and stores
// (a warp per column, lanes along its rows); the substitution runs one thread
// per column.  X has a padded row stride so both access patterns are
// conflict-free.
template <typename C2>
__global__ void lu_trsm_kernel(C2* A, long long lda, long long strideA, int n, int k, int kb, int c_begin, int c_end) {
  extern __shared__ unsigned char smem_raw[];
  C2* L = reinterpret_cast<C2*>(smem_raw);  // kb x kb, column-major
  C2* X = L + kb * kb;                      // kb x (blockDim + 1)
  const int ldx = blockDim.x + 1;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  C2* M = A + (size_t)blockIdx.y * strideA;
  for (int i = threadIdx.x; i < kb * kb; i += blockDim.x) {
    const int r = i % kb, c = i / kb;
    L[i] = M[(size_t)(k + c) * lda + k + r];
  }
  const int c0 = c_begin + blockIdx.x * blockDim.x;
  const int ncol = min((int)blockDim.x, c_end - c0);
  // 8 columns x 2 row halves per warp and batch: 16 independent loads in flight
  for (int cb = wid; cb < ncol; cb += 8 * nw) {
    C2 v[8][2];
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cl = cb + u * nw, r = lane + 32 * h;
        if (cl < ncol && r < kb) v[u][h] = M[(size_t)(c0 + cl) * lda + k + r];
      }
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cl = cb + u * nw, r = lane + 32 * h;
        if (cl < ncol && r < kb) X[r * ldx + cl] = v[u][h];
      }
  }
  __syncthreads();
  if ((int)threadIdx.x < ncol) {
    const int t = threadIdx.x;
    for (int j = 0; j < kb; ++j) {
      const C2 xj = X[j * ldx + t];
      for (int i = j + 1; i < kb; ++i) {
        const C2 l = L[j * kb + i];
        C2 v = X[i * ldx + t];
        v.x -= l.x * xj.x - l.y * xj.y;
        v.y -= l.x * xj.y + l.y * xj.x;
        X[i * ldx + t] = v;
      }
    }
  }
  __syncthreads();
  for (int cl = wid; cl < ncol; cl += nw) {
    C2* dst = M + (size_t)(c0 + cl) * lda + k;
    for (int r = lane; r < kb; r += 32) dst[r] = X[r * ldx + cl];
  }
}

// The FP64 form's U rows of a full panel: X = L11^{-1} X for 32 columns per CTA.  Each
// quarter of an SM has half an FP64 lane per clock, so one instruction of one warp takes 64
// cycles and four warps of a CTA work at once: warp w keeps rows w, w + 4, .. of its 32
// columns in registers (lane = column), the rows' new values go through shared memory, one
// barrier per row.  A thread per column left three quarters of each SM idle and waited for
// its shared-memory stores (the compiler cannot tell L from X).
// Two matrices of order 1,994, 32 rows: 157 -> 23 us (64 rows took 500).  With the panels
// of 32 the factorisation of both takes 56.4 ms where it took 81.5 (35 are the products at
// the FP64 pipe's rate); 16 of order 642: 24.6 -> 16.4 ms.  One level of 32-deep products is
// faster than two levels of 64, 128 or 256 (65.1 against 68.7, 70.5 and 71.2 ms before the
// triangular solve's change): cuBLAS loses more on the skinny shapes inside an outer block.
template <int KB>
__global__ void __launch_bounds__(128) lu_trsm64_kernel(double2* A, long long lda, long long strideA, int k,
                                                        int c_begin, int c_end) {
  extern __shared__ unsigned char smem_raw[];
  double2* L = reinterpret_cast<double2*>(smem_raw);  // KB x KB, column-major
  double2* X = L + KB * KB;                           // KB x 33
  constexpr int ldx = 33, RW = KB / 4;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2* M = A + (size_t)blockIdx.y * strideA;
  const int c0 = c_begin + blockIdx.x * 32;
  const int ncol = min(32, c_end - c0);
#pragma unroll 8
  for (int c = wid; c < KB; c += 4)
#pragma unroll
    for (int r = lane; r < KB; r += 32) L[c * KB + r] = M[(size_t)(k + c) * lda + k + r];
#pragma unroll 8
  for (int c = wid; c < 32; c += 4)
#pragma unroll
    for (int r = lane; r < KB; r += 32)
      X[r * ldx + c] = c < ncol ? M[(size_t)(c0 + c) * lda + k + r] : make_double2(0., 0.);
  __syncthreads();
  double2 v[RW];
#pragma unroll
  for (int q = 0; q < RW; ++q) v[q] = X[(4 * q + wid) * ldx + lane];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < KB; ++j) {
    if (wid == (j & 3)) X[j * ldx + lane] = v[j >> 2];
    __syncthreads();
    const double2 xj = X[j * ldx + lane];
#pragma unroll
    for (int q = j >> 2; q < RW; ++q) {
      if (q == (j >> 2) && wid <= (j & 3)) continue;
      const double2 l = L[j * KB + 4 * q + wid];
      v[q].x = fma(-l.x, xj.x, fma(l.y, xj.y, v[q].x));
      v[q].y = fma(-l.x, xj.y, fma(-l.y, xj.x, v[q].y));
    }
  }
  for (int c = wid; c < ncol; c += 4)
#pragma unroll
    for (int r = lane; r < KB; r += 32) M[(size_t)(c0 + c) * lda + k + r] = X[r * ldx + c];
}

template <int KB>
cudaError_t trsm64(double2* A, long long lda, long long strideA, int k, int c0, int c1, int batch, cudaStream_t stream) {
  constexpr size_t sm = (size_t)KB * (KB + 33) * sizeof(double2);
  if (sm > 32 * 1024) ensure_smem_limit((const void*)lu_trsm64_kernel<KB>, sm);
  dim3 g((unsigned)((c1 - c0 + 31) / 32), batch);
  lu_trsm64_kernel<KB><<<g, 128, sm, stream>>>(A, lda, strideA, k, c0, c1);
  return cudaGetLastError();
}

// The three steps around the 32-wide panels of the two-level LU (mixed form).  A panel of
// one matrix takes some tens of microseconds on at most 16 SMs, so what follows it has to
// be short as well; these kernels do the outer block's own part in plain FP32 FMAs, which
// a K = 32 product does in less time than it takes to split its operands for the tensor
// cores and read them back.  Measured at n = 4,976, one matrix (and 15): per 32 columns of
// the outer block, interchanges + U rows 6 us (29) where the two kernels before took 15,
// the rest of the block 7 us (30) where operand split + tcgen05 update took 13; per 256
// columns, the U rows for the trailing columns 40 us (310) where eight rounds of
// triangular solve, operand split and update took 180.  The time before was latency for
// one matrix (LU 16.9 -> 12.3 ms) and about the same work for 15 (75.7 -> 71.9 ms for 30).

// Applies a panel's net row permutation (rowmap) to every column outside the panel and
// turns rows k .. k + 31 of the outer block's columns right of it, [k + 32, c_end), into U
// rows: x = L11^{-1} x with the panel's unit lower triangle.  One warp per column.  The
// first `solve_ctas` CTAs take the columns to solve: lane = row of the diagonal block, its
// new value comes through shared memory, and the substitution broadcasts x_j from lane j.
// The others only permute; a warp more carries the row permutation so far (perm[i] =
// source of row i; null: none) as a column of its own.
__global__ void __launch_bounds__(256) lu_swap_urows_kernel(float2* A, long long lda, long long strideA, int n, int k,
                                                            int c_end, int solve_ctas,
                                                            const int* rowmap, int* perm) {
  __shared__ int sdst[128], ssrc[128];
  __shared__ float2 top[8][32];
  __shared__ float2 L[32][32];  // [column][row]
  __shared__ int s_cnt;
  const int* rm = rowmap + (size_t)blockIdx.y * kRowmapStride;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2* M = A + (size_t)blockIdx.y * strideA;
  const bool solver = (int)blockIdx.x < solve_ctas;
  grid_wait();
  grid_trigger();
  if (solver)
#pragma unroll
    for (int q = 0; q < 4; ++q) L[wid + 8 * q][lane] = M[(size_t)(k + wid + 8 * q) * lda + k + lane];
  if (threadIdx.x == 0) s_cnt = min(max(rm[0], 0), 128);
  __syncthreads();
  const int cnt = s_cnt;
  for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
    sdst[e] = rm[1 + 2 * e];
    ssrc[e] = rm[2 + 2 * e];
  }
  __syncthreads();
  if (solver) {
    const int c = k + 32 + blockIdx.x * 8 + wid;
    if (c >= c_end) return;
    float2* a = M + (size_t)c * lda;
    float2 v[4];
    top[wid][lane] = a[k + lane];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = lane + 32 * q;
      if (e < cnt && (unsigned)ssrc[e] < (unsigned)n) v[q] = a[ssrc[e]];
    }
    __syncwarp();  // every source is read before any destination is written
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = lane + 32 * q;
      if (e < cnt && (unsigned)ssrc[e] < (unsigned)n && (unsigned)sdst[e] < (unsigned)n) {
        if ((unsigned)(sdst[e] - k) < 32u)
          top[wid][sdst[e] - k] = v[q];
        else
          a[sdst[e]] = v[q];
      }
    }
    __syncwarp();
    float2 x = top[wid][lane];
#pragma unroll
    for (int j = 0; j < 31; ++j) {
      const float xr = __shfl_sync(0xffffffffu, x.x, j), xi = __shfl_sync(0xffffffffu, x.y, j);
      const float2 l = L[j][lane];
      if (lane > j) {
        x.x = fmaf(-l.x, xr, fmaf(l.y, xi, x.x));
        x.y = fmaf(-l.x, xi, fmaf(-l.y, xr, x.y));
      }
    }
    a[k + lane] = x;
    return;
  }
  const int t = (blockIdx.x - solve_ctas) * 8 + wid;  // left of the panel, then right of the outer block
  const int rest = k + (n - c_end);
  if (cnt == 0 || t > rest) return;
  if (t < rest)
    permute_column(M + (size_t)(t < k ? t : c_end + (t - k)) * lda, n, cnt, sdst, ssrc);
  else if (perm != nullptr)
    permute_column(perm + (size_t)blockIdx.y * n, n, cnt, sdst, ssrc);
}

// A[r0 .. r0 + M, c0 .. c0 + N) -= A[r0 .., kc .. kc + 32) A[kc .. kc + 32, c0 ..): one CTA per
// 128 x 32 tile, both operands in shared memory, each thread 4 x 4 entries in registers
// (rows 32 apart, so every global access of a warp is one run of 256 bytes).
__global__ void __launch_bounds__(256) lu_update32_kernel(float2* A, long long lda, long long strideA, int r0, int M,
                                                          int c0, int N, int kc) {
  __shared__ float2 sl[32][128];
  __shared__ __align__(16) float2 su[32][32];
  float2* Mx = A + (size_t)blockIdx.z * strideA;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int row0 = blockIdx.x * 128, col0 = blockIdx.y * 32;
  grid_wait();
  grid_trigger();
  {
    const int r = tid & 127, kh = tid >> 7;
    const bool in = row0 + r < M;
    const float2* src = Mx + (size_t)kc * lda + r0 + row0 + r;
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = in ? src[(size_t)(2 * q + kh) * lda] : make_float2(0.f, 0.f);
    float2 u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int cc = col0 + wid + 8 * q;
      u[q] = cc < N ? Mx[(size_t)(c0 + cc) * lda + kc + lane] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) sl[2 * q + kh][r] = v[q];
#pragma unroll
    for (int q = 0; q < 4; ++q) su[lane][wid + 8 * q] = u[q];
  }
  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = row0 + lane + 32 * i, c = col0 + 4 * wid + j;
      acc[i][j] = r < M && c < N ? Mx[(size_t)(c0 + c) * lda + r0 + r] : make_float2(0.f, 0.f);
    }
  __syncthreads();
#pragma unroll 8
  for (int kk = 0; kk < 32; ++kk) {
    const float4 ua = *reinterpret_cast<const float4*>(&su[kk][4 * wid]);
    const float4 ub = *reinterpret_cast<const float4*>(&su[kk][4 * wid + 2]);
    const float2 u[4] = {make_float2(ua.x, ua.y), make_float2(ua.z, ua.w), make_float2(ub.x, ub.y),
                         make_float2(ub.z, ub.w)};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 l = sl[kk][lane + 32 * i];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j].x = fmaf(-l.x, u[j].x, fmaf(l.y, u[j].y, acc[i][j].x));
        acc[i][j].y = fmaf(-l.x, u[j].y, fmaf(-l.y, u[j].x, acc[i][j].y));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = row0 + lane + 32 * i, c = col0 + 4 * wid + j;
      if (r < M && c < N) Mx[(size_t)(c0 + c) * lda + r0 + r] = acc[i][j];
    }
}

// U rows of a whole outer block for the trailing columns: rows [k0, k0 + 256) of columns
// [c0, c1) become L^{-1} times themselves, L the unit lower triangle of the outer block.
// Left-looking over 32-row blocks: a warp owns CPW columns, lane = row of the current
// block; the block first takes its products with the solved blocks (their rows in the
// warp's shared memory, read as broadcasts), then the 32 x 32 substitution (x_j broadcast
// from lane j).  The CTA's warps walk the triangle's 36 tiles of 32 x 32 together, each
// tile staged once for all of them by asynchronous copies kUrowsStages - 1 tiles ahead
// (read directly by every warp, L's latency made the kernel four times slower).  CPW = 8
// needs the fewest shared-memory reads per FMA; 4 halves the time of a call whose columns
// leave SMs idle.
constexpr int kUrowsWarps = 4, kUrowsStages = 4;
template <int CPW> constexpr size_t urows_smem() {
  return ((size_t)kUrowsStages * 32 * 32 + (size_t)kUrowsWarps * kOuterBlock * CPW) * sizeof(float2);
}
template <int CPW>
__global__ void __launch_bounds__(kUrowsWarps * 32) lu_urows_kernel(float2* A, long long lda, long long strideA, int k0,
                                                                    int c0, int c1) {
  constexpr int NBLK = kOuterBlock / 32, TILES = NBLK * (NBLK + 1) / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float2* ring = reinterpret_cast<float2*>(smem_raw);                                           // [stage][column][row]
  float2* X = ring + kUrowsStages * 32 * 32 + (size_t)wid * kOuterBlock * CPW;  // [row][CPW]
  float2* M = A + (size_t)blockIdx.y * strideA;
  const int cw = c0 + (blockIdx.x * kUrowsWarps + wid) * CPW;
  const int nc = max(0, min(CPW, c1 - cw));
  const float2* Lm = M + (size_t)k0 * lda + k0;
  int pb = 0, pl = 0;  // next tile to stage: rows 32 pb.., columns 32 pl..
  auto stage = [&](int slot) {
    if (pb < NBLK) {
      float2* dst = ring + (size_t)slot * 32 * 32;
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // 512 pieces of 16 bytes
        const int i = threadIdx.x + 128 * q, col = i >> 4, piece = i & 15;
        const float2* src = Lm + (size_t)(32 * pl + col) * lda + 32 * pb + 2 * piece;
        const unsigned d = (unsigned)__cvta_generic_to_shared(dst + 32 * col + 2 * piece);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src));
      }
      if (++pl > pb) {
        pl = 0;
        ++pb;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  grid_wait();
  for (int i = 0; i < kUrowsStages - 1; ++i) stage(i);
  float2 x[CPW], nx[CPW];  // the current block's rows, and the next one's
#pragma unroll
  for (int c = 0; c < CPW; ++c) nx[c] = c < nc ? M[(size_t)(cw + c) * lda + k0 + lane] : make_float2(0.f, 0.f);
  int b = 0, l = 0;
  for (int t = 0; t < TILES; ++t) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kUrowsStages - 2) : "memory");
    __syncthreads();  // tile t is in place for every warp, and tile t - 1 is no longer read
    stage((t + kUrowsStages - 1) % kUrowsStages);
    const float2* T = ring + (size_t)(t % kUrowsStages) * 32 * 32 + lane;
    if (l == 0) {
#pragma unroll
      for (int c = 0; c < CPW; ++c) x[c] = nx[c];
      if (b + 1 < NBLK) {
#pragma unroll
        for (int c = 0; c < CPW; ++c)
          nx[c] = c < nc ? M[(size_t)(cw + c) * lda + k0 + 32 * (b + 1) + lane] : make_float2(0.f, 0.f);
      }
    }
    if (l < b) {
      const float4* xs = reinterpret_cast<const float4*>(X + (size_t)32 * l * CPW);
#pragma unroll 8
      for (int kk = 0; kk < 32; ++kk) {
        const float2 lv = T[32 * kk];
#pragma unroll
        for (int q = 0; q < CPW / 2; ++q) {
          const float4 u = xs[kk * (CPW / 2) + q];
          x[2 * q].x = fmaf(-lv.x, u.x, fmaf(lv.y, u.y, x[2 * q].x));
          x[2 * q].y = fmaf(-lv.x, u.y, fmaf(-lv.y, u.x, x[2 * q].y));
          x[2 * q + 1].x = fmaf(-lv.x, u.z, fmaf(lv.y, u.w, x[2 * q + 1].x));
          x[2 * q + 1].y = fmaf(-lv.x, u.w, fmaf(-lv.y, u.z, x[2 * q + 1].y));
        }
      }
      ++l;
    } else {
#pragma unroll
      for (int j = 0; j < 31; ++j) {
        const float2 lv = T[32 * j];
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
          const float xr = __shfl_sync(0xffffffffu, x[c].x, j), xi = __shfl_sync(0xffffffffu, x[c].y, j);
          if (lane > j) {
            x[c].x = fmaf(-lv.x, xr, fmaf(lv.y, xi, x[c].x));
            x[c].y = fmaf(-lv.x, xi, fmaf(-lv.y, xr, x[c].y));
          }
        }
      }
      float4* xd = reinterpret_cast<float4*>(X + (size_t)(32 * b + lane) * CPW);
#pragma unroll
      for (int q = 0; q < CPW / 2; ++q) xd[q] = make_float4(x[2 * q].x, x[2 * q].y, x[2 * q + 1].x, x[2 * q + 1].y);
      __syncwarp();
#pragma unroll
      for (int c = 0; c < CPW; ++c)
        if (c < nc) M[(size_t)(cw + c) * lda + k0 + 32 * b + lane] = x[c];
      l = 0;
      ++b;
    }
  }
}

__global__ void iota_rows_kernel(int* __restrict__ perm, int n, int total) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total) perm[i] = i % n;
}

__global__ void f64_to_f32_kernel(const double2* s, float2* d, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) d[i] = make_float2((float)s[i].x, (float)s[i].y);
}

}  // namespace

bool tc_gemm_plan(TcGemmPlan* p, void* workspace, int n, int batch, float2* A, long long lda, int nb);
cudaError_t tc_trailing_update(TcGemmPlan* p, float2* A, long long lda, long long strideA, int n, int k, int kb,
                               cudaStream_t stream);
cudaError_t tc_update(TcGemmPlan* p, float2* A, long long lda, long long strideA, int row0, int M, int col0, int N,
                      int kcol0, int K, cudaStream_t stream);
size_t tc_gemm_plan_size();

namespace {

// State of one batched factorisation for the two-level driver (mixed form).
struct LuJob {
  float2* A;
  long long lda, strideA;
  int n, batch, nb, cl;
  int* ipiv;
  int* info;
  int* rowmap;
  int* perm;         // row permutation of the whole factorisation, built panel by panel (null: not wanted)
  TcGemmPlan* plan;  // tcgen05 updates
  cudaStream_t stream;
  int polls;         // of the panels' exchange
  int rule_batch;
};

// U rows [k, k+kb) of columns [c0, c1): U = L^{-1} A with L the unit lower triangle of A[k:k+kb, k:k+kb].
cudaError_t trsm_cols(const LuJob& j, int k, int kb, int c0, int c1) {
  if (c1 <= c0 || kb <= 0) return cudaSuccess;
  const int tpb = 128;
  dim3 g((unsigned)((c1 - c0 + tpb - 1) / tpb), j.batch);
  const size_t sm = (size_t)kb * kb * sizeof(float2) + (size_t)kb * (tpb + 1) * sizeof(float2);
  if (sm > 48 * 1024) ensure_smem_limit((const void*)lu_trsm_kernel<float2>, sm);
  lu_trsm_kernel<float2><<<g, tpb, sm, j.stream>>>(j.A, j.lda, j.strideA, j.n, k, kb, c0, c1);
  return cudaGetLastError();
}

// A[r0:r0+M, c0:c0+N] -= A[r0:r0+M, kc:kc+K] * A[kc:kc+K, c0:c0+N] for every matrix.
cudaError_t block_update(const LuJob& j, int r0, int M, int c0, int N, int kc, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return cudaSuccess;
  return tc_update(j.plan, j.A, j.lda, j.strideA, r0, M, c0, N, kc, K, j.stream);
}

#define BEM_TRY(x)                          \
  do {                                      \
    const cudaError_t e_ = (x);             \
    if (e_ != cudaSuccess) return e_;       \
  } while (0)

// U rows of outer block k0 (kOuterBlock wide) for columns [c0, c1).
cudaError_t outer_urows(const LuJob& j, int k0, int c0, int c1) {
  auto run = [&](auto cpw_c) {
    constexpr int CPW = decltype(cpw_c)::value;
    constexpr size_t sm = urows_smem<CPW>();
    ensure_smem_limit((const void*)lu_urows_kernel<CPW>, sm);
    dim3 g((unsigned)((c1 - c0 + kUrowsWarps * CPW - 1) / (kUrowsWarps * CPW)), j.batch);
    return launch_chained(lu_urows_kernel<CPW>, g, kUrowsWarps * 32, sm, j.stream, j.A, j.lda, j.strideA, k0,
                          c0, c1);
  };
  // 8 columns per warp where that still gives every SM a CTA, else 4
  const long long cols = (long long)(c1 - c0) * j.batch;
  if (cols >= 8LL * kUrowsWarps * sm_count()) return run(std::integral_constant<int, 8>{});
  return run(std::integral_constant<int, 4>{});
}

// Columns of the next outer block when `rest` are left.  The boundary of an outer block (U
// rows, operand split, tensor-core update) takes about 65 us of latency, so the last ones
// are taken as one block, whose FP32 updates cost less: up to 1,024 columns of one matrix,
// fewer of a batch, whose updates fill the GPU (about 2.5 million entries in all), and 512
// at any batch.  LU before and after: order 520, one matrix 0.68 -> 0.59 ms, 16 0.84 ->
// 0.80; order 998, one 1.79 -> 1.67, 16 2.40 -> 2.38 (2.82 as one block); order 1,520, one
// 2.83 -> 2.64.
int outer_width(int rest, int NB, int batch, bool narrow) {
  if (narrow && (rest <= 2 * NB || (rest <= 4 * NB && (long long)rest * rest * batch <= 2500000))) return rest;
  return std::min(NB, rest);
}

// Two-level right-looking LU.  The matrix is factored in outer block columns of
// width NB (kOuterBlock, 256): each is factored as sub-panels of width nb (the cluster panel
// width, 32 or 64) with their row interchanges applied to every other column
// and the rest of the outer block updated after each sub-panel; then the outer
// block's U rows are solved and the trailing matrix takes one
// update of depth NB.  The trailing matrix is read and written once per NB
// columns instead of once per nb, which at block depth 64 bounds the LU by HBM.
// Sub-panels of 32 columns (the mixed form's) take the three FP32 kernels above; 64-wide
// ones (options.lu_block) the general triangular solve and updates.
// Panel, swap + U rows and update follow one another three times per 32 columns, each a few
// microseconds long, so they are chained launches: the next one's CTAs are in place, and
// the panel's exchange slots cleared, when the one before ends (LU of one matrix of order
// 498: 0.77 -> 0.68 ms; 4,976: 11.7 -> 11.1; 16 of 498: 0.89 -> 0.85).  The panel triggers
// its successor after its last step, so that no waiting CTA holds an SM of another stream.
cudaError_t lu_two_level(const LuJob& j, int NB) {
  const int n = j.n, nb = j.nb;
  const bool narrow = nb == 32;
  if (j.perm) {
    const int total = n * j.batch;
    iota_rows_kernel<<<(total + 255) / 256, 256, 0, j.stream>>>(j.perm, n, total);
  }
  for (int k0 = 0, KB; k0 < n; k0 += KB) {
    KB = outer_width(n - k0, NB, j.rule_batch, narrow);
    for (int j0 = 0; j0 < KB; j0 += nb) {
      const int kb = std::min(nb, KB - j0), kk = k0 + j0;
      BEM_TRY(lu_panel_cluster(Precision::Mixed, j.A, j.lda, j.strideA, n, kk, kb, nb, j.cl, j.batch, j.ipiv, j.info, j.stream,
                               j.rowmap, j.polls));
      if (narrow && kb == 32) {
        const int rest = k0 + KB - kk - 32;  // the rest of the outer block
        const int solve_ctas = (rest + 7) / 8;
        dim3 gs((unsigned)(solve_ctas + (kk + n - k0 - KB + (j.perm ? 1 : 0) + 7) / 8), j.batch);
        if (gs.x > 0)
          BEM_TRY(launch_chained(lu_swap_urows_kernel, gs, 256, 0, j.stream, j.A, j.lda, j.strideA, n, kk, k0 + KB,
                                 solve_ctas, j.rowmap, j.perm));
        if (rest > 0) {
          dim3 gu((unsigned)((n - kk - 32 + 127) / 128), (unsigned)((rest + 31) / 32), j.batch);
          BEM_TRY(launch_chained(lu_update32_kernel, gu, 256, 0, j.stream, j.A, j.lda, j.strideA, kk + 32, n - kk - 32,
                                 kk + 32, rest, kk));
        }
        BEM_TRY(cudaGetLastError());
        continue;
      }
      BEM_TRY(lu_swap_rows_batched(Precision::Mixed, j.A, j.lda, j.strideA, n, kk, kb, j.batch, j.rowmap, j.perm, j.stream));
      if (j0 + kb < KB) {  // the rest of the outer block
        BEM_TRY(trsm_cols(j, kk, kb, kk + kb, k0 + KB));
        BEM_TRY(block_update(j, kk + kb, n - kk - kb, kk + kb, k0 + KB - kk - kb, kk, kb));
      }
    }
    if (k0 + KB < n) {
      if (narrow) {
        BEM_TRY(outer_urows(j, k0, k0 + KB, n));
      } else {
        // U rows of the outer block for the trailing columns: blocked forward substitution
        for (int i0 = 0; i0 < KB; i0 += nb) {
          const int kb = std::min(nb, KB - i0), kk = k0 + i0;
          BEM_TRY(trsm_cols(j, kk, kb, k0 + KB, n));
          if (i0 + kb < KB) BEM_TRY(block_update(j, kk + kb, k0 + KB - kk - kb, k0 + KB, n - k0 - KB, kk, kb));
        }
      }
      BEM_TRY(block_update(j, k0 + KB, n - k0 - KB, k0 + KB, n - k0 - KB, k0, KB));
    }
  }
  return cudaGetLastError();
}

}  // namespace

int lu_launch_count(int n, int nb, int NB, bool perm, int batch) {
  const int per_update = 2;  // operand split + tcgen05 kernel
  const bool narrow = nb == 32;
  int count = perm ? 1 : 0;
  for (int k0 = 0, KB; k0 < n; k0 += KB) {
    KB = outer_width(n - k0, NB, batch, narrow);
    for (int j0 = 0; j0 < KB; j0 += nb) {
      const int kb = std::min(nb, KB - j0);
      count += 2;                                        // panel, row swaps (narrow: with the U rows)
      if (j0 + kb < KB) count += narrow ? 1 : 1 + (n - k0 - j0 - kb > 0 ? per_update : 0);
    }
    if (k0 + KB < n) {
      if (narrow)
        count += 1;
      else
        for (int i0 = 0; i0 < KB; i0 += nb) count += 1 + (i0 + std::min(nb, KB - i0) < KB ? per_update : 0);
      count += per_update;
    }
  }
  return count;
}

cudaError_t lu_factor_batched(Precision prec, void* A, long long lda, int n, int batch, int* ipiv, int* info, int nb,
                              void* cublas_handle, cudaStream_t stream, LuGemm gemm, void* tc_workspace,
                              bool* used_tensor, int** tc_err, int* rowmap, int* n_launches, int* perm, int polls,
                              int rule_batch) {
  if (rule_batch <= 0) rule_batch = batch;
  cublasHandle_t h = (cublasHandle_t)cublas_handle;
  cublasSetStream(h, stream);
  const long long strideA = lda * (long long)n;
  const bool mixed = prec == Precision::Mixed;
  const int want_nb = (nb == 32 || nb == 64) ? nb : 0;  // 0: automatic
  nb = nb > 0 ? std::min(nb, 64) : (mixed ? 64 : 32);
  const size_t esz = mixed ? sizeof(float2) : sizeof(double2);
  int cnb = 0, ccl = 0;
  const bool cluster_panel = lu_cluster_plan(prec, n, want_nb, batch, &cnb, &ccl);
  if (cluster_panel) nb = cnb;
  // tensor-core trailing update (mixed precision only; K = 2 nb <= 128)
  std::vector<unsigned char> plan_storage;
  TcGemmPlan* plan = nullptr;
  if (mixed && gemm != LuGemm::Cublas && tc_workspace && nb <= 64 && tc_gemm_available()) {
    plan_storage.resize(tc_gemm_plan_size());
    plan = reinterpret_cast<TcGemmPlan*>(plan_storage.data());
    if (!tc_gemm_plan(plan, tc_workspace, n, batch, (float2*)A, lda, nb)) plan = nullptr;
  }
  if (gemm == LuGemm::Tensor && mixed && !plan) return cudaErrorNotSupported;
  if (used_tensor) *used_tensor = plan != nullptr;
  if (plan) {
    if (tc_err) *tc_err = tc_gemm_error_word(plan);
    cudaMemsetAsync(tc_gemm_error_word(plan), 0, sizeof(int), stream);
  }
  // The two-level schedule serves the HBM-bound tcgen05 update; cuBLAS (the FP64
  // form, or lu_gemm = 1) keeps one level: its kernels for the skinny panel
  // shapes of the two-level schedule are slow.
  if (cluster_panel && rowmap && plan) {
    LuJob job{(float2*)A, lda, strideA, n, batch, nb, ccl, ipiv, info, rowmap, perm, plan, stream, polls, rule_batch};
    if (n_launches) *n_launches = lu_launch_count(n, nb, kOuterBlock, perm != nullptr, rule_batch);
    return lu_two_level(job, kOuterBlock);
  }
  if (n_launches) *n_launches = 0;
  for (int k = 0; k < n; k += nb) {
    const int kb = std::min(nb, n - k);
    if (n_launches) *n_launches += 2 + (n - k - kb > 0 ? 1 + (plan ? 2 : 0) : 0);
    if (cluster_panel) {
      cudaError_t e = lu_panel_cluster(prec, A, lda, strideA, n, k, kb, nb, ccl, batch, ipiv, info, stream, rowmap, polls);
      if (e != cudaSuccess) return e;
    } else if (mixed)
      lu_panel_kernel<float><<<batch, 1024, 0, stream>>>((float2*)A, lda, strideA, n, k, kb, ipiv, info);
    else
      lu_panel_kernel<double><<<batch, 1024, 0, stream>>>((double2*)A, lda, strideA, n, k, kb, ipiv, info);
    if (n - kb > 0 && cluster_panel && rowmap) {
      cudaError_t e = lu_swap_rows_batched(prec, A, lda, strideA, n, k, kb, batch, rowmap, nullptr, stream);
      if (e != cudaSuccess) return e;
    } else if (n - kb > 0) {
      dim3 g((n - kb + 127) / 128, batch);
      if (mixed)
        lu_swap_kernel<float2><<<g, 128, 0, stream>>>((float2*)A, lda, strideA, n, k, kb, ipiv);
      else
        lu_swap_kernel<double2><<<g, 128, 0, stream>>>((double2*)A, lda, strideA, n, k, kb, ipiv);
    }
    const int rest = n - k - kb;
    if (rest > 0) {
      const int tpb = 128;
      dim3 g((rest + tpb - 1) / tpb, batch);
      const size_t sm = (size_t)kb * kb * esz + (size_t)kb * (tpb + 1) * esz;
      if (mixed) {
        if (sm > 48 * 1024) ensure_smem_limit((const void*)lu_trsm_kernel<float2>, sm);
        lu_trsm_kernel<float2><<<g, tpb, sm, stream>>>((float2*)A, lda, strideA, n, k, kb, k + kb, n);
        if (plan) {
          cudaError_t e = tc_trailing_update(plan, (float2*)A, lda, strideA, n, k, kb, stream);
          if (e != cudaSuccess) return e;
          continue;
        }
        const cuComplex alpha = make_cuComplex(-1.f, 0.f), beta = make_cuComplex(1.f, 0.f);
        float2* base = (float2*)A;
        cublasStatus_t st = cublasCgemmStridedBatched(
            h, CUBLAS_OP_N, CUBLAS_OP_N, rest, rest, kb, &alpha, (const cuComplex*)(base + (k + kb) + (size_t)k * lda),
            (int)lda, strideA, (const cuComplex*)(base + k + (size_t)(k + kb) * lda), (int)lda, strideA, &beta,
            (cuComplex*)(base + (k + kb) + (size_t)(k + kb) * lda), (int)lda, strideA, batch);
        if (st != CUBLAS_STATUS_SUCCESS) return cudaErrorUnknown;
      } else {
        if (kb == 32 || kb == 64) {
          const cudaError_t e = kb == 32 ? trsm64<32>((double2*)A, lda, strideA, k, k + kb, n, batch, stream)
                                         : trsm64<64>((double2*)A, lda, strideA, k, k + kb, n, batch, stream);
          if (e != cudaSuccess) return e;
        } else {
          if (sm > 48 * 1024) ensure_smem_limit((const void*)lu_trsm_kernel<double2>, sm);
          lu_trsm_kernel<double2><<<g, tpb, sm, stream>>>((double2*)A, lda, strideA, n, k, kb, k + kb, n);
        }
        const cuDoubleComplex alpha = make_cuDoubleComplex(-1.0, 0.0), beta = make_cuDoubleComplex(1.0, 0.0);
        double2* base = (double2*)A;
        cublasStatus_t st = cublasZgemmStridedBatched(
            h, CUBLAS_OP_N, CUBLAS_OP_N, rest, rest, kb, &alpha,
            (const cuDoubleComplex*)(base + (k + kb) + (size_t)k * lda), (int)lda, strideA,
            (const cuDoubleComplex*)(base + k + (size_t)(k + kb) * lda), (int)lda, strideA, &beta,
            (cuDoubleComplex*)(base + (k + kb) + (size_t)(k + kb) * lda), (int)lda, strideA, batch);
        if (st != CUBLAS_STATUS_SUCCESS) return cudaErrorUnknown;
      }
    }
  }
  if (perm) {
    if (n_launches) *n_launches += 1;
    return lu_perm_batched(ipiv, n, batch, perm, stream);
  }
  return cudaGetLastError();
}

cudaError_t convert_f64_to_f32(const double2* src, float2* dst, long long n, cudaStream_t stream) {
  f64_to_f32_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(src, dst, n);
  return cudaGetLastError();
}

}  // namespace bem
