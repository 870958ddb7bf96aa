// Cluster-resident LU panel factorisation and cluster triangular solves (sm_103a).
//
// Panels: lu_panel_reg_kernel (mixed form) and lu_panel_reg64_kernel (FP64 form) keep a row
// of 32 columns per thread in registers and exchange pivot candidates as tagged words
// (described at the kernels); they serve every order whose rows fit a cluster of 16.
// lu_panel_cluster_kernel takes the rest (64-wide panels, partial last panels, larger
// orders): the m x nb panel of one matrix is spread over the shared memory of a
// thread-block cluster (CL CTAs, each holding a contiguous block of panel rows,
// column-major).  Each column step does a local pivot search, publishes the
// CTA's candidate row, one cluster barrier, a pivot decision from the CL
// candidates read through distributed shared memory (DSMEM), then the swap,
// scaling and rank-1 update entirely in shared memory.
// Pivot choice is LAPACK's (first maximum of |re| + |im|) in all three.
//
// Solves (FP64 form, and orders whose rows bem_lu_solve.cu cannot hold): each right-hand
// side is solved by one cluster whose CTAs own blocks of rows: the owner of a 32-row
// diagonal block solves it with one warp, publishes the 32 values in a double-buffered
// shared slot, and after one cluster barrier every CTA applies the block's
// columns to its own rows.
//
// Cluster barriers are hardware barriers (barrier.cluster); every CTA of a
// cluster executes the same sequence of them, and the kernels end with a
// barrier so no CTA leaves while another may still read its shared memory.
#include <cooperative_groups.h>
#include <limits.h>

#include <array>
#include <map>
#include <mutex>
#include <type_traits>

#include "bem_common.cuh"
#include "bem_kernels.h"

namespace cg = cooperative_groups;

namespace bem {
namespace {

template <typename R> struct CT2;
template <> struct CT2<float> { typedef float2 C2; };
template <> struct CT2<double> { typedef double2 C2; };

template <typename C2> __device__ __forceinline__ auto abs1(C2 v) -> decltype(v.x) { return fabs(v.x) + fabs(v.y); }

constexpr int kPanelThreads = 512;

// First maximum of (value, index): larger value wins, ties go to the smaller index
// (LAPACK's first maximum of |re| + |im| when indices are row numbers).
template <typename R> __device__ __forceinline__ void argmax_merge(R& b, int& x, R ov, int oi) {
  if (ov > b || (ov == b && oi < x)) {
    b = ov;
    x = oi;
  }
}
template <typename R> __device__ __forceinline__ void warp_argmax(R& b, int& x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) argmax_merge(b, x, __shfl_xor_sync(0xffffffffu, b, o), __shfl_xor_sync(0xffffffffu, x, o));
}

// Net row permutation of the interchanges (j, pivs[j]), j = 0..kb-1, applied in
// order (LAPACK laswp): row r of every column ends up holding the data of row
// src(r).  Computed by one warp: the rows of the diagonal block in top[], other
// pivot rows in a list searched with a ballot.  Writes [count, (k + r, k + src(r))
// for every moved row] (at most 2 kb pairs).
template <int NB> __device__ void net_row_map(const int* pivs, int kb, int k, int* out) {
  __shared__ int top[NB], erow[NB], econt[NB];
  const int lane = threadIdx.x & 31;
  for (int i = lane; i < kb; i += 32) top[i] = i;
  __syncwarp();
  int n_ext = 0;
  for (int j = 0; j < kb; ++j) {
    const int p = pivs[j];
    if (p == j) continue;
    if (p < kb) {
      if (lane == 0) {
        const int t = top[j];
        top[j] = top[p];
        top[p] = t;
      }
      __syncwarp();
      continue;
    }
    int found = -1;
    for (int base = 0; base < n_ext && found < 0; base += 32) {
      const int idx = base + lane;
      const unsigned hit = __ballot_sync(0xffffffffu, idx < n_ext && erow[idx] == p);
      if (hit) found = base + __ffs(hit) - 1;
    }
    if (found < 0) {
      found = n_ext++;
      if (lane == 0) {
        erow[found] = p;
        econt[found] = p;
      }
    }
    __syncwarp();
    if (lane == 0) {
      const int t = top[j];
      top[j] = econt[found];
      econt[found] = t;
    }
    __syncwarp();
  }
  if (lane == 0) {
    int cnt = 0;
    for (int r = 0; r < kb; ++r)
      if (top[r] != r) {
        out[1 + 2 * cnt] = k + r;
        out[2 + 2 * cnt] = k + top[r];
        ++cnt;
      }
    for (int e = 0; e < n_ext; ++e)
      if (econt[e] != erow[e]) {
        out[1 + 2 * cnt] = k + erow[e];
        out[2 + 2 * cnt] = k + econt[e];
        ++cnt;
      }
    out[0] = cnt;
  }
}

// Apply a net row permutation to the columns outside the panel, one warp per column.  One
// warp more does the same to the row permutation so far (perm, null: none).
template <typename C2>
__global__ void __launch_bounds__(256) lu_swap_rows_kernel(C2* A, long long lda, long long strideA, int n, int k,
                                                          int kb, const int* rowmap, int* perm) {
  __shared__ int sdst[128], ssrc[128];
  __shared__ int s_cnt;
  const int* rm = rowmap + (size_t)blockIdx.y * kRowmapStride;
  if (threadIdx.x == 0) s_cnt = min(max(rm[0], 0), 128);
  __syncthreads();
  const int cnt = s_cnt;
  for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
    sdst[e] = rm[1 + 2 * e];
    ssrc[e] = rm[2 + 2 * e];
  }
  __syncthreads();
  const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (cnt == 0 || t > n - kb) return;
  if (t < n - kb)
    permute_column(A + (size_t)blockIdx.y * strideA + (size_t)(t < k ? t : t + kb) * lda, n, cnt, sdst, ssrc);
  else if (perm != nullptr)
    permute_column(perm + (size_t)blockIdx.y * n, n, cnt, sdst, ssrc);
}

// One column step has a single cluster barrier.  Before it, every CTA
// publishes its local pivot candidate (value, row) and the candidate's whole
// panel row, and the owner of row j publishes row j, into slot j & 1.  After
// it, every CTA reads the CL candidates (one lane each), takes the first
// maximum, copies the winning row and row j from their owners' slots, and
// finishes the column locally.  A slot is rewritten two columns later, after
// the next barrier, by which time every CTA has finished reading it.
template <typename R, int NB>
__global__ void __launch_bounds__(kPanelThreads) lu_panel_cluster_kernel(typename CT2<R>::C2* A, long long lda,
                                                                         long long strideA, int n, int k, int kb,
                                                                         int chunk, int* ipiv, int* info,
                                                                         int* rowmap) {
  typedef typename CT2<R>::C2 C2;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int CL = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int NW = blockDim.x >> 5;
  __shared__ int s_pivs[NB];  // pivot row of each column, panel-local (rank 0)
  C2* M = A + (size_t)blockIdx.y * strideA;
  int* piv = ipiv + (size_t)blockIdx.y * n;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2* P = reinterpret_cast<C2*>(smem_raw);  // [NB][chunk], this CTA's panel rows
  C2* pub = P + (size_t)NB * chunk;         // [2][NB] published candidate row
  C2* dg = pub + 2 * NB;                    // [2][NB] published row j (owner of row j)
  C2* urow = dg + 2 * NB;                   // pivot row after the interchange
  C2* drow = urow + NB;                     // row j before the interchange
  R* cval = reinterpret_cast<R*>(drow + NB);         // [2] published candidate value
  int* cidx = reinterpret_cast<int*>(cval + 2);      // [2] published candidate row
  __shared__ R wval[32];
  __shared__ int widx[32];
  __shared__ int s_bi, s_p, s_fallback;

  const int m = n - k;
  const int r0 = rank * chunk;
  const int rows = max(0, min(chunk, m - r0));
  // panel load: each thread owns rows, 16 independent column loads in flight
  for (int i = tid; i < rows; i += blockDim.x) {
    const C2* src = M + (size_t)k * lda + k + r0 + i;
#pragma unroll 16
    for (int c = 0; c < NB; ++c)
      if (c < kb) P[(size_t)c * chunk + i] = src[(size_t)c * lda];
  }
  __syncthreads();

  for (int j = 0; j < kb; ++j) {
    const int s = j & 1;
    const int owner_j = j / chunk;
    // local pivot candidate among this CTA's panel rows >= j
    R best = R(-1);
    int bi = INT_MAX;
    const C2* Pj = P + (size_t)j * chunk;
    for (int i = max(0, j - r0) + tid; i < rows; i += blockDim.x) argmax_merge(best, bi, abs1(Pj[i]), r0 + i);
    warp_argmax(best, bi);
    if (lane == 0) {
      wval[wid] = best;
      widx[wid] = bi;
    }
    __syncthreads();
    if (wid == 0) {
      R b = lane < NW ? wval[lane] : R(-1);
      int x = lane < NW ? widx[lane] : INT_MAX;
      warp_argmax(b, x);
      if (lane == 0) {
        cval[s] = b;
        cidx[s] = x;
        s_bi = x;
      }
    }
    __syncthreads();
    const int bi_loc = s_bi;
    if (bi_loc != INT_MAX)
      for (int c = tid; c < kb; c += blockDim.x) pub[s * NB + c] = P[(size_t)c * chunk + (bi_loc - r0)];
    if (rank == owner_j)
      for (int c = tid; c < kb; c += blockDim.x) dg[s * NB + c] = P[(size_t)c * chunk + (j - r0)];
    cluster.sync();  // candidates, candidate rows and row j of this column are published
    if (wid == 0) {
      R b = R(-1);
      int x = INT_MAX;
      if (lane < CL) {
        b = *cluster.map_shared_rank(cval + s, lane);
        x = *cluster.map_shared_rank(cidx + s, lane);
      }
      warp_argmax(b, x);
      if (lane == 0) {
        s_fallback = x == INT_MAX;  // no comparable candidate (all NaN): keep row j
        s_p = x == INT_MAX ? j : x;
      }
    }
    __syncthreads();
    const int p = s_p;
    const int owner_p = p / chunk;
    {
      const C2* src_u = s_fallback ? cluster.map_shared_rank(dg + s * NB, owner_j)
                                   : cluster.map_shared_rank(pub + s * NB, owner_p);
      const C2* src_d = cluster.map_shared_rank(dg + s * NB, owner_j);
      for (int c = tid; c < kb; c += blockDim.x) {
        urow[c] = src_u[c];
        drow[c] = src_d[c];
      }
    }
    __syncthreads();
    if (p != j) {
      if (rank == owner_j)
        for (int c = tid; c < kb; c += blockDim.x) P[(size_t)c * chunk + (j - r0)] = urow[c];
      if (rank == owner_p)
        for (int c = tid; c < kb; c += blockDim.x) P[(size_t)c * chunk + (p - r0)] = drow[c];
    }
    if (rank == 0 && tid == 0) {
      piv[k + j] = k + p;
      s_pivs[j] = p;
    }
    __syncthreads();
    const C2 d = urow[j];
    C2 inv;
    if (d.x == R(0) && d.y == R(0)) {
      inv.x = R(0);
      inv.y = R(0);
      if (rank == 0 && tid == 0 && info[blockIdx.y] == 0) info[blockIdx.y] = k + j + 1;
    } else {
      inv = pivot_inverse<true>(d);
    }
    const int i0 = min(rows, max(0, j + 1 - r0));  // first local row below the diagonal
    C2* Pcol = P + (size_t)j * chunk;
    for (int i = i0 + tid; i < rows; i += blockDim.x) Pcol[i] = cmul(Pcol[i], inv);
    __syncthreads();
    // rank-1 update of columns j+1.. : warps take columns, lanes take rows
    for (int c = j + 1 + wid; c < kb; c += NW) {
      const C2 u = urow[c];
      C2* Pc = P + (size_t)c * chunk;
      for (int i = i0 + lane; i < rows; i += 32) {
        const C2 l = Pcol[i];
        C2 v = Pc[i];
        v.x -= l.x * u.x - l.y * u.y;
        v.y -= l.x * u.y + l.y * u.x;
        Pc[i] = v;
      }
    }
    __syncthreads();
  }
  for (int i = tid; i < rows; i += blockDim.x) {
    C2* dst = M + (size_t)k * lda + k + r0 + i;
#pragma unroll 16
    for (int c = 0; c < NB; ++c)
      if (c < kb) dst[(size_t)c * lda] = P[(size_t)c * chunk + i];
  }
  if (rank == 0 && wid == 0 && rowmap != nullptr) net_row_map<NB>(s_pivs, kb, k, rowmap + (size_t)blockIdx.y * kRowmapStride);
  cluster.sync();  // no CTA leaves while others may still read its shared memory
}

// Register-resident panel (mixed form, 32 columns): one thread per panel row.
// The thread keeps the part of its row right of the current column in
// registers, shifted so that the current column is always a[0] (every register
// index is a constant, and the step loop stays rolled); the multipliers it
// produces go to shared memory (Lb[column][thread]).  Interchanges are virtual:
// each thread carries the logical row index lg of its physical row, the pivot
// search compares logical indices (LAPACK's first maximum of |re| + |im|), and
// every row is written once, at the end, to its logical position, which is also
// the net row permutation that the other columns get.  A step:
//  1. every warp takes this CTA's candidate from the warps' keys; the warp that
//     holds the candidate row copies it from its thread's registers through a
//     shared row and pushes it with the key into slot j & 1 of every CTA (DSMEM);
//  2. every 64-bit word pushed carries the step's number beside its 32 bits of
//     payload, so the receivers poll their own shared memory for it: no fence, no
//     cluster barrier, one DSMEM store's latency per step.  A slot is rewritten at
//     step j + 2, by a CTA that has seen every CTA's step j + 1, which those push
//     after the barrier that ends their reading of step j;
//  3. every warp takes the pivot from the CTAs' keys, waits for the pivot row
//     (columns j.. as u[0..]) and lays it out for broadcast reads; rank 0 stores it;
//  4. the pivot row leaves (lg = j), the row with lg = j takes the pivot's old
//     lg; every other active row stores l = a[0] / pivot, subtracts l u and
//     shifts; the next candidate is reduced per warp; CTA barrier.
// The polls are bounded (`polls` reads of a word): a CTA that waits in vain leaves its
// panel without storing its rows, and info = -1 and an empty row map say so.  No place in
// memory is computed from words that did not all arrive.
// A single CTA (CLUSTER = false) replaces 1 and 2 by the owner thread writing the
// row to its own shared memory and a CTA barrier.
// Requires a full panel (kb = 32) and chunk <= kRegPanelThreads.
//
// Bound: the latency of a column step (the candidate exchange, one CTA barrier and the row
// update, about 440 issue cycles with 640 rows on an SM).  The keys are reduced by the
// warp-reduction instruction (two 32-bit maxima instead of five 64-bit shuffle stages),
// one warp instead of 640 threads does the push, and no row-j copy is kept for the
// all-NaN case (a NaN key ranks below every number, so row j itself wins it): 32 columns
// of one matrix took 74 us, then 29 us with one CTA (518 rows) and 53 us with eight (4,976)
// exchanging through a fence and a cluster barrier, 49 us through tagged words.
constexpr int kRegPanelThreads = 640;
constexpr int kRegPanelWarps = kRegPanelThreads / 32;

// Pivot candidates as two 32-bit words, compared as (hi, lo): the bits of |re| + |im|
// plus one (non-negative floats order as their bits; 0 for NaN) and the complement of the
// logical row, so the largest key is the first maximum (larger value, then smaller row).
// A row that is no candidate has (0, 0), below every candidate: lo >= 2^31 for any row.
__device__ __forceinline__ uint2 pivot_key(float v, int row) {
  return make_uint2(v == v ? __float_as_uint(v) + 1u : 0u, (unsigned)~row);
}
__device__ __forceinline__ uint2 warp_max_key(uint2 k) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, k.x);
  return make_uint2(hi, __reduce_max_sync(0xffffffffu, k.x == hi ? k.y : 0u));
}

// Words of the exchange: 32 bits of payload with the step's tag above them, written and read
// whole (64-bit accesses are single-copy atomic).  Keys pack (hi, lo): lo's 16 low bits are
// those of ~row (rows < 10,240; 0 only where there is no candidate), its high ones the tag.
__device__ __forceinline__ void push_words(void* dst, unsigned long long a, unsigned long long b) {
  asm volatile("st.relaxed.cluster.v2.b64 [%0], {%1, %2};" ::"l"(dst), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void push_word(void* dst, unsigned long long a) {
  asm volatile("st.relaxed.cluster.b64 [%0], %1;" ::"l"(dst), "l"(a) : "memory");
}
__device__ __forceinline__ unsigned long long poll_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.cluster.shared::cta.b64 %0, [%1];"
               : "=l"(v)
               : "r"((unsigned)__cvta_generic_to_shared(p))
               : "memory");
  return v;
}
__device__ __forceinline__ ulonglong2 poll_words(const unsigned long long* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.cluster.shared::cta.v2.b64 {%0, %1}, [%2];"
               : "=l"(v.x), "=l"(v.y)
               : "r"((unsigned)__cvta_generic_to_shared(p))
               : "memory");
  return v;
}

template <bool CLUSTER>
__global__ void __launch_bounds__(kRegPanelThreads, 1) lu_panel_reg_kernel(float2* A, long long lda, long long strideA,
                                                                           int n, int k, int kb, int chunk, int* ipiv,
                                                                           int* info, int* rowmap, int polls) {
  constexpr int NB = 32;
  constexpr int NW = kRegPanelWarps;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = CLUSTER ? (int)cluster.block_rank() : 0;
  const int CL = CLUSTER ? (int)cluster.num_blocks() : 1;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float2* Lb = reinterpret_cast<float2*>(smem_raw);  // [NB][kRegPanelThreads] multipliers by column, thread
  __shared__ __align__(16) unsigned long long rowsT[2][CLUSTER ? 16 : 1][2 * NB];  // pushed rows (tagged re, im), by source CTA
  __shared__ unsigned long long keyT[2][16];                                      // pushed keys, by source CTA
  __shared__ __align__(16) float4 urow[2][NB / 2];  // the pivot row for broadcast reads (CLUSTER: [0]; else by step parity)
  __shared__ __align__(16) float4 pub[NB / 2];
  __shared__ uint2 wkey[2][NW];  // by step parity
  // this CTA gave up waiting, by step parity: a warp that reads it behind the barrier of step j
  // must not see what a faster one writes in step j + 1
  __shared__ int s_failed[2];
  __shared__ int s_any_failed;  // any CTA did (rank 0's)
  __shared__ int s_moved;       // rows that changed place (rank 0's counts for the cluster)
  float2* M = A + (size_t)blockIdx.y * strideA;
  int* piv = ipiv + (size_t)blockIdx.y * n;
  const int m = n - k;
  const int r0 = rank * chunk;
  const int rows = max(0, min(chunk, m - r0));
  const bool mine = tid < rows;
  int lg = r0 + tid;         // logical row of this thread's physical row
  int done_at = -1;          // step at which this row became the pivot row
  if (tid == 0) {
    s_moved = 0;
    s_failed[0] = s_failed[1] = 0;
    s_any_failed = 0;
  }
  if constexpr (CLUSTER) {  // no tag of an earlier use in the slots when the first push arrives
    for (int i = tid; i < 2 * 16 * 2 * NB; i += kRegPanelThreads) (&rowsT[0][0][0])[i] = 0ull;
    if (tid < 32) (&keyT[0][0])[tid] = 0ull;
    cluster.sync();
  }
  grid_wait();
  float2 a[NB];
  {
    const float2* src = M + (size_t)k * lda + k + r0 + tid;
#pragma unroll
    for (int c = 0; c < NB; ++c) a[c] = mine ? src[(size_t)c * lda] : make_float2(0.f, 0.f);
  }
  auto publish_warp_key = [&](int parity) {  // the warp's candidate for the current column
    const uint2 key = warp_max_key(mine && done_at < 0 ? pivot_key(abs1(a[0]), lg) : make_uint2(0u, 0u));
    if (lane == 0) wkey[parity][wid] = key;
  };
  auto copy_row = [&](float4* dst) {
#pragma unroll
    for (int q = 0; q < NB / 2; ++q) dst[q] = make_float4(a[2 * q].x, a[2 * q].y, a[2 * q + 1].x, a[2 * q + 1].y);
  };
  publish_warp_key(0);
  __syncthreads();
#pragma unroll 1
  for (int j = 0; j < NB; ++j) {
    const int s = j & 1;
    const unsigned tag = (unsigned)(j + 1);
    // 1. this CTA's candidate, pushed by the warp that holds it
    uint2 key = warp_max_key(lane < NW ? wkey[s][lane] : make_uint2(0u, 0u));
    const bool own = mine && done_at < 0 && key.y != 0u && lg == (int)~key.y;  // logical rows are distinct
    if constexpr (CLUSTER) {
      const bool owner_warp = __ballot_sync(0xffffffffu, own) != 0u;
      // the key first: every CTA can decide while the rows are still on their way
      if ((owner_warp || (key.y == 0u && wid == 0)) && lane < CL)  // without a candidate row, warp 0 says so
        push_word(cluster.map_shared_rank(&keyT[s][rank], lane),
                  ((unsigned long long)key.x << 32) | (tag << 16) | (key.y & 0xffffu));
      if (owner_warp) {
        if (own) copy_row(pub);
        __syncwarp();
        const float2 v = reinterpret_cast<const float2*>(pub)[lane];
        const unsigned long long wr = ((unsigned long long)tag << 32) | __float_as_uint(v.x);
        const unsigned long long wi = ((unsigned long long)tag << 32) | __float_as_uint(v.y);
#pragma unroll 4
        for (int t = 0; t < CL; ++t) push_words(cluster.map_shared_rank(&rowsT[s][rank][2 * lane], t), wr, wi);
      }
    } else {
      if (own) copy_row(urow[s]);
      __syncthreads();
    }
    // 3. pivot (logical row p, held by CTA pr), in every warp; row j itself is a candidate, so there is one
    const float4* U = urow[CLUSTER ? 0 : s];  // the pivot row, u[c] = U(j, j + c) (zero beyond the panel)
    int p = (int)~key.y;
    if constexpr (CLUSTER) {
      unsigned long long kw = 0ull;
      bool ok;
      int left = polls;
      do {  // the bound's test below the read: on top, LU of one matrix of order 4,976 took 11.3 ms, here 10.7
        if (lane < CL) kw = poll_word(&keyT[s][lane]);
        ok = __all_sync(0xffffffffu, lane >= CL || ((unsigned)kw >> 16) == tag);
      } while (!ok && --left > 0);
      const uint2 ck = lane < CL ? make_uint2((unsigned)(kw >> 32), (unsigned)kw & 0xffffu) : make_uint2(0u, 0u);
      key = warp_max_key(ck);
      const int pr = __ffs(__ballot_sync(0xffffffffu, ck.x == key.x && ck.y == key.y)) - 1;  // keys are distinct
      p = (int)(~key.y & 0xffffu);
      ulonglong2 u = make_ulonglong2(0ull, 0ull);
      bool got;
      left = polls;
      do {
        u = poll_words(&rowsT[s][pr][2 * lane]);
        got = __all_sync(0xffffffffu, (unsigned)(u.x >> 32) == tag && (unsigned)(u.y >> 32) == tag);
      } while (!got && --left > 0);
      if (!(ok && got) || polls == 0) s_failed[s] = 1;  // this warp's p is worth nothing: no row is stored
      // every warp writes the same values; the barrier that ends the step keeps step j + 1's away
      reinterpret_cast<float2*>(urow[0])[lane] = make_float2(__uint_as_float((unsigned)u.x), __uint_as_float((unsigned)u.y));
      __syncwarp();
    }
    if (rank == 0 && wid == 0 && lane < NB - j)  // U row j
      M[(size_t)(k + j + lane) * lda + k + j] = reinterpret_cast<const float2*>(U)[lane];
    if (rank == 0 && tid == 0) piv[k + j] = k + p;
    const float2 d = make_float2(U[0].x, U[0].y);
    // whether |d|^2 is in range is known from the key, before the row arrives
    const bool plain = key.x - __float_as_uint(0x1p-49f) <= __float_as_uint(0x1p49f) - __float_as_uint(0x1p-49f);
    const float2 inv = plain ? pivot_inverse_plain<false>(d) : pivot_inverse_scaled<false>(d);
    if (rank == 0 && tid == 0 && d.x == 0.f && d.y == 0.f && info[blockIdx.y] == 0) info[blockIdx.y] = k + j + 1;
    // 4. this thread's row
    if (mine && done_at < 0) {
      if (lg == p) {  // the pivot row: it is logical row j now, finished
        lg = j;
        done_at = j;
      } else {
        if (lg == j) lg = p;  // the old row j moves to the pivot's place
        const float2 l = cmul(a[0], inv);
        Lb[(size_t)j * kRegPanelThreads + tid] = l;
        // a[c - 1] = a[c] - l u[c] for columns j + 1.. .  From step j the window holds 32 - j
        // live columns, so the update runs over the smallest multiple of 8 covering them (the
        // columns beyond are zero).  (Packed FP32x2 FMAs on a duplicated copy of the pivot
        // row took 4 more registers than the 96 a 640-thread CTA allows and spilled.)
        auto update = [&](auto width) {
          constexpr int W = decltype(width)::value;
#pragma unroll
          for (int q = 0; q < W / 2; ++q) {
            const float4 u = U[q];
            if (q > 0) {
              a[2 * q - 1].x = fmaf(-l.x, u.x, fmaf(l.y, u.y, a[2 * q].x));
              a[2 * q - 1].y = fmaf(-l.x, u.y, fmaf(-l.y, u.x, a[2 * q].y));
            }
            a[2 * q].x = fmaf(-l.x, u.z, fmaf(l.y, u.w, a[2 * q + 1].x));
            a[2 * q].y = fmaf(-l.x, u.w, fmaf(-l.y, u.z, a[2 * q + 1].y));
          }
          a[W - 1] = make_float2(0.f, 0.f);
        };
        if (j < 8)
          update(std::integral_constant<int, 32>{});
        else if (j < 16)
          update(std::integral_constant<int, 24>{});
        else if (j < 24)
          update(std::integral_constant<int, 16>{});
        else
          update(std::integral_constant<int, 8>{});
      }
    }
    publish_warp_key(s ^ 1);
    __syncthreads();
    if (CLUSTER && s_failed[s]) break;  // uniform in the CTA; the other CTAs wait in vain in turn
  }
  grid_trigger();
  const bool failed = CLUSTER && (s_failed[0] | s_failed[1]);
  if (CLUSTER && failed && tid == 0) *cluster.map_shared_rank(&s_any_failed, 0) = 1;
  // every row to its logical position: the multipliers left of its pivot column
  // (all 32 for rows that never became the pivot)
  if (mine && !failed) {
    const int ncol = done_at < 0 ? NB : done_at;
    float2* dst = M + (size_t)k * lda + k + lg;
    for (int c = 0; c < ncol; ++c) dst[(size_t)c * lda] = Lb[(size_t)c * kRegPanelThreads + tid];
  }
  // the net row permutation, [count, (dst row, src row) x count] in any order (at most 2 kb rows move)
  if (rowmap != nullptr) {
    int* rm = rowmap + (size_t)blockIdx.y * kRowmapStride;
    if (mine && !failed && lg != r0 + tid) {
      const int e = atomicAdd(CLUSTER ? cluster.map_shared_rank(&s_moved, 0) : &s_moved, 1);
      rm[1 + 2 * e] = k + lg;
      rm[2 + 2 * e] = k + r0 + tid;
    }
    if constexpr (!CLUSTER) __syncthreads();
  }
  if constexpr (CLUSTER) cluster.sync();  // no CTA leaves while others may still use its shared memory
  if (rank == 0 && tid == 0) {
    const bool gave_up = CLUSTER && s_any_failed;
    if (gave_up) info[blockIdx.y] = -1;
    if (rowmap != nullptr) rowmap[(size_t)blockIdx.y * kRowmapStride] = gave_up ? 0 : s_moved;
  }
}

// The register-resident panel of the FP64 form: the algorithm of lu_panel_reg_kernel with
// the row's 32 complex doubles in 128 registers (256 threads), always on a cluster.  What
// differs:
//  - pivot keys are three words, (hi, lo) of |re| + |im| plus one in hi, and the complement
//    of the logical row: the same first maximum, exactly;
//  - the pivot's reciprocal is formed by the owner's thread and pushed behind the row: with
//    two FP64 lanes per SM an instruction of one warp takes 16 cycles of the pipe, so the
//    two divisions in every warp would cost more than the rest of the step's overhead;
//  - the cluster is as wide as the batch leaves room for (choose_panel): the row update is
//    bound by the FP64 pipe, 2 lanes per SM and clock, not by latency alone.
// Two matrices of order 1,994: 64 columns in two panels of 156 us on 2 x 16 SMs, where the
// shared-memory panel of 64 took 775 us.  Of a step's 4.9 us the row update is 2.4 us (one
// warp per quarter of an SM), exchange and reciprocal the rest.
constexpr int kReg64Threads = 256;
constexpr int kReg64Warps = kReg64Threads / 32;

__device__ __forceinline__ uint3 pivot_key64(double v, int row) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  return v == v ? make_uint3(hi + 1u, lo, (unsigned)~row) : make_uint3(0u, 0u, (unsigned)~row);
}
__device__ __forceinline__ uint3 warp_max_key(uint3 k) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, k.x);
  const unsigned lo = __reduce_max_sync(0xffffffffu, k.x == hi ? k.y : 0u);
  return make_uint3(hi, lo, __reduce_max_sync(0xffffffffu, k.x == hi && k.y == lo ? k.z : 0u));
}
__device__ __forceinline__ unsigned long long tagged(unsigned tag, int word) {
  return ((unsigned long long)tag << 32) | (unsigned)word;
}
__device__ __forceinline__ double untagged(ulonglong2 w) { return __hiloint2double((int)(unsigned)w.x, (int)(unsigned)w.y); }

__global__ void __launch_bounds__(kReg64Threads, 1) lu_panel_reg64_kernel(double2* A, long long lda, long long strideA,
                                                                          int n, int k, int kb, int chunk, int* ipiv,
                                                                          int* info, int* rowmap, int polls) {
  constexpr int NB = 32;
  constexpr int NW = kReg64Warps;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), CL = (int)cluster.num_blocks();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* Lb = reinterpret_cast<double2*>(smem_raw);  // [NB][kReg64Threads] multipliers by column, thread
  // pushed rows by source CTA, (hi, lo) of re and im per column, then the reciprocal
  __shared__ __align__(16) unsigned long long rowsT[2][16][4 * (NB + 1)];
  __shared__ __align__(16) unsigned long long keyT[2][16][2];  // pushed keys, by source CTA
  __shared__ __align__(16) double2 pub[NB + 1];                // the candidate row and its reciprocal
  __shared__ __align__(16) double2 urow[NB + 1];               // the pivot row and its reciprocal
  __shared__ uint3 wkey[2][NW];                                // by step parity
  // this CTA gave up waiting, by step parity: a warp that reads it behind the barrier of step j
  // must not see what a faster one writes in step j + 1
  __shared__ int s_failed[2];
  __shared__ int s_any_failed;  // any CTA did (rank 0's)
  __shared__ int s_moved;       // rows that changed place (rank 0's counts for the cluster)
  double2* M = A + (size_t)blockIdx.y * strideA;
  int* piv = ipiv + (size_t)blockIdx.y * n;
  const int m = n - k;
  const int r0 = rank * chunk;
  const int rows = max(0, min(chunk, m - r0));
  const bool mine = tid < rows;
  int lg = r0 + tid;  // logical row of this thread's physical row
  int done_at = -1;   // step at which this row became the pivot row
  double2 a[NB];
  {
    const double2* src = M + (size_t)k * lda + k + r0 + tid;
#pragma unroll
    for (int c = 0; c < NB; ++c) a[c] = mine ? src[(size_t)c * lda] : make_double2(0., 0.);
  }
  auto publish_warp_key = [&](int parity) {  // the warp's candidate for the current column
    const uint3 key = warp_max_key(mine && done_at < 0 ? pivot_key64(abs1(a[0]), lg) : make_uint3(0u, 0u, 0u));
    if (lane == 0) wkey[parity][wid] = key;
  };
  if (tid == 0) {
    s_moved = 0;
    s_failed[0] = s_failed[1] = 0;
    s_any_failed = 0;
  }
  publish_warp_key(0);
  // no tag of an earlier use in the slots when the first push arrives
  for (int i = tid; i < 2 * 16 * 4 * (NB + 1); i += kReg64Threads) (&rowsT[0][0][0])[i] = 0ull;
  if (tid < 64) (&keyT[0][0][0])[tid] = 0ull;
  cluster.sync();
#pragma unroll 1
  for (int j = 0; j < NB; ++j) {
    const int s = j & 1;
    const unsigned tag = (unsigned)(j + 1);
    // 1. this CTA's candidate, pushed by the warp that holds it, the key first
    uint3 key = warp_max_key(lane < NW ? wkey[s][lane] : make_uint3(0u, 0u, 0u));
    const bool own = mine && done_at < 0 && key.z != 0u && lg == (int)~key.z;  // logical rows are distinct
    const bool owner_warp = __ballot_sync(0xffffffffu, own) != 0u;
    if ((owner_warp || (key.z == 0u && wid == 0)) && lane < CL)  // without a candidate row, warp 0 says so
      push_words(cluster.map_shared_rank(&keyT[s][rank][0], lane),
                 ((unsigned long long)key.x << 32) | (tag << 16) | (key.z & 0xffffu),
                 ((unsigned long long)key.y << 32) | tag);
    if (owner_warp) {
      if (own) {
#pragma unroll
        for (int q = 0; q < NB; ++q) pub[q] = a[q];
        pub[NB] = pivot_inverse(a[0]);
      }
      __syncwarp();
      for (int c = lane; c < NB + 1; c += 32) {
        const double2 v = pub[c];
        const unsigned long long w0 = tagged(tag, __double2hiint(v.x)), w1 = tagged(tag, __double2loint(v.x));
        const unsigned long long w2 = tagged(tag, __double2hiint(v.y)), w3 = tagged(tag, __double2loint(v.y));
#pragma unroll 4
        for (int t = 0; t < CL; ++t) {
          unsigned long long* dst = cluster.map_shared_rank(&rowsT[s][rank][4 * c], t);
          push_words(dst, w0, w1);
          push_words(dst + 2, w2, w3);
        }
      }
    }
    // 2. pivot (logical row p, held by CTA pr), in every warp; row j itself is a candidate, so there is one
    ulonglong2 kw = make_ulonglong2(0ull, 0ull);
    bool ok;
    int left = polls;
    do {
      if (lane < CL) kw = poll_words(&keyT[s][lane][0]);
      ok = __all_sync(0xffffffffu, lane >= CL || (((unsigned)kw.x >> 16) == tag && (unsigned)kw.y == tag));
    } while (!ok && --left > 0);
    const uint3 ck = lane < CL ? make_uint3((unsigned)(kw.x >> 32), (unsigned)(kw.y >> 32), (unsigned)kw.x & 0xffffu)
                               : make_uint3(0u, 0u, 0u);
    key = warp_max_key(ck);
    const int pr = __ffs(__ballot_sync(0xffffffffu, ck.x == key.x && ck.y == key.y && ck.z == key.z)) - 1;  // distinct
    const int p = (int)(~key.z & 0xffffu);
    bool got;
    left = polls;
    do {
      const unsigned long long* src = rowsT[s][pr];
      const ulonglong2 re = poll_words(src + 4 * lane), im = poll_words(src + 4 * lane + 2);
      const ulonglong2 ire = poll_words(src + 4 * NB), iim = poll_words(src + 4 * NB + 2);
      auto here = [&](ulonglong2 w) { return (unsigned)(w.x >> 32) == tag && (unsigned)(w.y >> 32) == tag; };
      got = __all_sync(0xffffffffu, here(re) && here(im) && here(ire) && here(iim));
      // every warp writes the same values; the barrier that ends the step keeps step j + 1's away
      if (got) {
        urow[lane] = make_double2(untagged(re), untagged(im));
        if (lane == 0) urow[NB] = make_double2(untagged(ire), untagged(iim));
      }
    } while (!got && --left > 0);
    if (!(ok && got) || polls == 0) s_failed[s] = 1;
    __syncwarp();
    if (rank == 0 && wid == 0 && lane < NB - j) M[(size_t)(k + j + lane) * lda + k + j] = urow[lane];  // U row j
    if (rank == 0 && tid == 0) {
      piv[k + j] = k + p;
      if (urow[0].x == 0. && urow[0].y == 0. && info[blockIdx.y] == 0) info[blockIdx.y] = k + j + 1;
    }
    // 3. this thread's row
    if (mine && done_at < 0) {
      if (lg == p) {  // the pivot row: it is logical row j now, finished
        lg = j;
        done_at = j;
      } else {
        if (lg == j) lg = p;  // the old row j moves to the pivot's place
        const double2 l = cmul(a[0], urow[NB]);
        Lb[(size_t)j * kReg64Threads + tid] = l;
        // a[c - 1] = a[c] - l u[c] for columns j + 1.., over the smallest multiple of 4 that
        // covers the 32 - j live columns (the columns beyond are zero)
        auto update = [&](auto width) {
          constexpr int W = decltype(width)::value;
#pragma unroll
          for (int c = 1; c < W; ++c) {
            const double2 u = urow[c];
            a[c - 1].x = fma(-l.x, u.x, fma(l.y, u.y, a[c].x));
            a[c - 1].y = fma(-l.x, u.y, fma(-l.y, u.x, a[c].y));
          }
          a[W - 1] = make_double2(0., 0.);
        };
        switch (j >> 2) {
          case 0: update(std::integral_constant<int, 32>{}); break;
          case 1: update(std::integral_constant<int, 28>{}); break;
          case 2: update(std::integral_constant<int, 24>{}); break;
          case 3: update(std::integral_constant<int, 20>{}); break;
          case 4: update(std::integral_constant<int, 16>{}); break;
          case 5: update(std::integral_constant<int, 12>{}); break;
          case 6: update(std::integral_constant<int, 8>{}); break;
          default: update(std::integral_constant<int, 4>{}); break;
        }
      }
    }
    publish_warp_key(s ^ 1);
    __syncthreads();
    if (s_failed[s]) break;  // uniform in the CTA; the other CTAs wait in vain in turn
  }
  const bool failed = s_failed[0] | s_failed[1];
  if (failed && tid == 0) *cluster.map_shared_rank(&s_any_failed, 0) = 1;
  // every row to its logical position: the multipliers left of its pivot column
  // (all 32 for rows that never became the pivot)
  if (mine && !failed) {
    const int ncol = done_at < 0 ? NB : done_at;
    double2* dst = M + (size_t)k * lda + k + lg;
    for (int c = 0; c < ncol; ++c) dst[(size_t)c * lda] = Lb[(size_t)c * kReg64Threads + tid];
  }
  if (rowmap != nullptr && mine && !failed && lg != r0 + tid) {  // the net row permutation, as above
    int* rm = rowmap + (size_t)blockIdx.y * kRowmapStride;
    const int e = atomicAdd(cluster.map_shared_rank(&s_moved, 0), 1);
    rm[1 + 2 * e] = k + lg;
    rm[2 + 2 * e] = k + r0 + tid;
  }
  cluster.sync();  // no CTA leaves while others may still use its shared memory
  if (rank == 0 && tid == 0) {
    if (s_any_failed) info[blockIdx.y] = -1;
    if (rowmap != nullptr) rowmap[(size_t)blockIdx.y * kRowmapStride] = s_any_failed ? 0 : s_moved;
  }
}

// perm[i] such that (P b)[i] = b[perm[i]], from LAPACK-style interchanges.
__global__ void lu_perm_kernel(const int* __restrict__ ipiv, int n, int* __restrict__ perm) {
  extern __shared__ int sp[];
  const int* piv = ipiv + (size_t)blockIdx.x * n;
  int* out = perm + (size_t)blockIdx.x * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) sp[i] = i;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 0; i < n; ++i) {
      const int p = piv[i];
      if (p != i && p >= 0 && p < n) {
        const int t = sp[i];
        sp[i] = sp[p];
        sp[p] = t;
      }
    }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = sp[i];
}

constexpr int kSolveThreads = 512;

// One cluster per (matrix, right-hand side): x = U^{-1} L^{-1} (P b), in place in B.
// Pull rows [lo, hi) of columns [c0, c0 + 32) of M (column-major, clipped to
// the n x n matrix) into L2 ahead of their use: one prefetch per 128-byte line,
// spread over the CTA's threads.
template <typename C2>
__device__ __forceinline__ void prefetch_strip_l2(const C2* M, long long lda, int n, int c0, int lo, int hi) {
  constexpr int kPerLine = 128 / (int)sizeof(C2);
  lo = max(lo, 0);
  hi = min(hi, n);
  if (hi <= lo || c0 >= n) return;
  const int first = lo / kPerLine, last = (hi - 1) / kPerLine;
  const int lines = last - first + 1;
  const int cols = min(32, n - c0);
  for (int i = threadIdx.x; i < lines * cols; i += blockDim.x) {
    const int c = i / lines, l = i - c * lines;
    const C2* ptr = M + (size_t)(c0 + c) * lda + (size_t)(first + l) * kPerLine;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr));
  }
}

template <typename R>
__global__ void __launch_bounds__(kSolveThreads) lu_solve_cluster_kernel(const typename CT2<R>::C2* A, long long lda,
                                                                         long long strideA, int n,
                                                                         const int* __restrict__ perm,
                                                                         typename CT2<R>::C2* B, long long ldb,
                                                                         int nrhs, int chunk) {
  typedef typename CT2<R>::C2 C2;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31;
  const int sys = blockIdx.y;
  const int mat = sys / nrhs;
  const C2* M = A + (size_t)mat * strideA;
  C2* b = B + (size_t)sys * ldb;
  const int* pm = perm + (size_t)mat * n;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2* x = reinterpret_cast<C2*>(smem_raw);  // my rows [r0, r0 + chunk)
  C2* pub = x + chunk;                      // [2][32] published block solutions
  const int r0 = rank * chunk;
  const int rows = max(0, min(chunk, n - r0));
  for (int i = tid; i < rows; i += blockDim.x) x[i] = b[pm[r0 + i]];
  cluster.sync();  // every CTA has read b before anyone writes it back
  const int nblk = (n + 31) / 32;
  // forward substitution with unit lower L
  if (rows > 0) prefetch_strip_l2(M, lda, n, 0, r0, r0 + rows);
  for (int t = 0; t < nblk; ++t) {
    const int k0 = t * 32, kb = min(32, n - k0);
    const int owner = k0 / chunk;
    C2* slot = pub + 32 * (t & 1);
    // the next step's columns of my rows (its diagonal block included) stream into L2 meanwhile
    if (rows > 0 && t + 1 < nblk) prefetch_strip_l2(M, lda, n, k0 + 32, max(r0, k0 + 32), r0 + rows);
    if (rank == owner && tid < 32) {
      // this lane's row of the diagonal block, loaded up front (independent loads)
      C2 Lr[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (j < kb && lane < kb) {
          Lr[j] = M[(size_t)(k0 + j) * lda + k0 + lane];
        } else {
          Lr[j].x = 0;
          Lr[j].y = 0;
        }
      }
      C2 v;
      v.x = 0;
      v.y = 0;
      if (lane < kb) v = x[k0 - r0 + lane];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        C2 xj;
        xj.x = __shfl_sync(0xffffffffu, v.x, j);
        xj.y = __shfl_sync(0xffffffffu, v.y, j);
        if (lane > j) {
          v.x -= Lr[j].x * xj.x - Lr[j].y * xj.y;
          v.y -= Lr[j].x * xj.y + Lr[j].y * xj.x;
        }
      }
      if (lane < kb) {
        x[k0 - r0 + lane] = v;
        slot[lane] = v;
      }
    }
    cluster.sync();
    __shared__ C2 xs[32];
    if (tid < kb) xs[tid] = cluster.map_shared_rank(slot, owner)[tid];
    __syncthreads();
    for (int i = tid; i < rows; i += blockDim.x) {
      const int r = r0 + i;
      if (r < k0 + kb) continue;
      C2 v = x[i];
      if (sizeof(C2) == sizeof(float2) && kb == 32) {  // FP32: all 32 loads in flight at once
        C2 l[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) l[j] = M[(size_t)(k0 + j) * lda + r];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const C2 s = xs[j];
          v.x -= l[j].x * s.x - l[j].y * s.y;
          v.y -= l[j].x * s.y + l[j].y * s.x;
        }
      } else {
#pragma unroll 8
        for (int j = 0; j < kb; ++j) {
          const C2 l = M[(size_t)(k0 + j) * lda + r];
          const C2 s = xs[j];
          v.x -= l.x * s.x - l.y * s.y;
          v.y -= l.x * s.y + l.y * s.x;
        }
      }
      x[i] = v;
    }
    __syncthreads();
  }
  // backward substitution with U
  if (rows > 0) prefetch_strip_l2(M, lda, n, (nblk - 1) * 32, r0, min(r0 + rows, n));
  for (int t = nblk - 1; t >= 0; --t) {
    const int k0 = t * 32, kb = min(32, n - k0);
    const int owner = k0 / chunk;
    // the next (lower) block's columns of my rows above its diagonal block's end
    if (rows > 0 && t > 0) prefetch_strip_l2(M, lda, n, k0 - 32, r0, min(r0 + rows, k0));
    // the slot alternates over the whole sequence of blocks (forward then backward)
    C2* slot = pub + 32 * ((nblk + (nblk - 1 - t)) & 1);
    if (rank == owner && tid < 32) {
      C2 Ur[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (j < kb && lane < kb) {
          Ur[j] = M[(size_t)(k0 + j) * lda + k0 + lane];
        } else {
          Ur[j].x = 0;
          Ur[j].y = 0;
        }
      }
      C2 dinv;
      dinv.x = 0;
      dinv.y = 0;
      if (lane < kb) dinv = pivot_inverse<true>(M[(size_t)(k0 + lane) * lda + k0 + lane]);
      C2 v;
      v.x = 0;
      v.y = 0;
      if (lane < kb) v = x[k0 - r0 + lane];
#pragma unroll
      for (int j = 31; j >= 0; --j) {
        if (lane == j) v = cmul(v, dinv);
        C2 xj;
        xj.x = __shfl_sync(0xffffffffu, v.x, j);
        xj.y = __shfl_sync(0xffffffffu, v.y, j);
        if (lane < j) {
          v.x -= Ur[j].x * xj.x - Ur[j].y * xj.y;
          v.y -= Ur[j].x * xj.y + Ur[j].y * xj.x;
        }
      }
      if (lane < kb) {
        x[k0 - r0 + lane] = v;
        slot[lane] = v;
      }
    }
    cluster.sync();
    __shared__ C2 ys[32];
    if (tid < kb) ys[tid] = cluster.map_shared_rank(slot, owner)[tid];
    __syncthreads();
    for (int i = tid; i < rows; i += blockDim.x) {
      const int r = r0 + i;
      if (r >= k0) continue;
      C2 v = x[i];
      if (sizeof(C2) == sizeof(float2) && kb == 32) {  // FP32: all 32 loads in flight at once
        C2 u[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) u[j] = M[(size_t)(k0 + j) * lda + r];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const C2 s = ys[j];
          v.x -= u[j].x * s.x - u[j].y * s.y;
          v.y -= u[j].x * s.y + u[j].y * s.x;
        }
      } else {
#pragma unroll 8
        for (int j = 0; j < kb; ++j) {
          const C2 u = M[(size_t)(k0 + j) * lda + r];
          const C2 s = ys[j];
          v.x -= u.x * s.x - u.y * s.y;
          v.y -= u.x * s.y + u.y * s.x;
        }
      }
      x[i] = v;
    }
    __syncthreads();
  }
  for (int i = tid; i < rows; i += blockDim.x) b[r0 + i] = x[i];
  cluster.sync();
}

template <typename K>
cudaError_t launch_cluster(K kern, dim3 grid, int threads, size_t smem, int cl, cudaStream_t stream,
                           void** args, bool chained = false) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained ? 2 : 1;  // chained: the kernel calls grid_wait
  return cudaLaunchKernelExC(&cfg, (const void*)kern, args);
}

// Largest cluster size the kernel can be launched with at this shared-memory size.
template <typename K> int max_cluster(K kern, int threads, size_t smem) {
  if (!ensure_smem_limit((const void*)kern, smem)) return 0;
  cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(16, 1);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  int cl = 0;
  if (cudaOccupancyMaxPotentialClusterSize(&cl, (const void*)kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return cl;
}

constexpr size_t kPanelSmemBudget = 200 * 1024;
constexpr size_t kReg64Smem = (size_t)32 * kReg64Threads * sizeof(double2);

template <typename R, int NB> size_t panel_smem(int chunk) {
  typedef typename CT2<R>::C2 C2;
  return (size_t)NB * chunk * sizeof(C2) + 6 * NB * sizeof(C2) + 64;
}

// Clusters of size cl that can be resident at once for this kernel and shared memory.
template <typename K> int active_clusters(K kern, int threads, size_t smem, int cl) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl, 1);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int num = 0;
  if (cudaOccupancyMaxActiveClusters(&num, (const void*)kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return num;
}

// Panel width and cluster size for an n x n batch.  The panel is latency-bound
// (an exchange between the cluster's CTAs per column), so the batch's panels should
// run in as few waves of clusters as possible: the register panel (32 wide) where its
// rows fit, else, among the (width, cluster size) pairs whose panel fits in shared
// memory, the fewest waves (batch / resident clusters), then the wider panel, then
// the smaller cluster.  want_nb > 0 fixes the width.
template <typename R> bool choose_panel(int n, int want_nb, int batch, int& nb, int& cl) {
  bool found = false;
  int best_waves = 0;
  if (sizeof(R) == 4 && (want_nb == 0 || want_nb == 32)) {
    // the register-resident panel (32 wide) where a cluster of at most 16 CTAs
    // holds the rows at one per thread: the fewest waves, then the smallest cluster
    for (int c : {1, 2, 4, 8, 16}) {
      if ((n + c - 1) / c > kRegPanelThreads) continue;
      const size_t sm = (size_t)32 * kRegPanelThreads * sizeof(float2);
      if (c > 1 && max_cluster(lu_panel_reg_kernel<true>, kRegPanelThreads, sm) < c) continue;
      if (c == 1 && !ensure_smem_limit((const void*)lu_panel_reg_kernel<false>, sm)) continue;
      const int act = c > 1 ? active_clusters(lu_panel_reg_kernel<true>, kRegPanelThreads, sm, c)
                            : active_clusters(lu_panel_reg_kernel<false>, kRegPanelThreads, sm, c);
      if (act < 1) continue;
      const int waves = (std::max(batch, 1) + act - 1) / act;
      if (!found || waves < best_waves) {
        found = true;
        best_waves = waves;
        nb = 32;
        cl = c;
      }
    }
    if (found) return true;
  }
  if (sizeof(R) == 8 && (want_nb == 0 || want_nb == 32)) {
    // the FP64 form's: a column step takes about 1.4 us of exchange and, at 2 FP64 lanes per
    // SM and clock, 20 ns per row of a CTA while all 32 columns are live (10 ns on average
    // over a factorisation's shrinking panels), so a wider cluster pays until it costs a wave
    double best = 0.0;
    for (int c : {2, 4, 8, 16}) {
      if ((n + c - 1) / c > kReg64Threads) continue;
      if (max_cluster(lu_panel_reg64_kernel, kReg64Threads, kReg64Smem) < c) continue;
      const int act = active_clusters(lu_panel_reg64_kernel, kReg64Threads, kReg64Smem, c);
      if (act < 1) continue;
      const double cost = (std::max(batch, 1) + act - 1) / act * (1.4 + 0.01 * n / c);
      if (!found || cost < best) {
        found = true;
        best = cost;
        nb = 32;
        cl = c;
      }
    }
    if (found) return true;
  }
  for (int w : {64, 32}) {
    if (want_nb > 0 && w != want_nb) continue;
    for (int c : {4, 8, 16}) {
      const int chunk = (n + c - 1) / c;
      const size_t sm = w == 64 ? panel_smem<R, 64>(chunk) : panel_smem<R, 32>(chunk);
      if (sm > kPanelSmemBudget) continue;
      const int maxcl = w == 64 ? max_cluster(lu_panel_cluster_kernel<R, 64>, kPanelThreads, sm)
                                : max_cluster(lu_panel_cluster_kernel<R, 32>, kPanelThreads, sm);
      if (maxcl < c) continue;
      const int act = w == 64 ? active_clusters(lu_panel_cluster_kernel<R, 64>, kPanelThreads, sm, c)
                              : active_clusters(lu_panel_cluster_kernel<R, 32>, kPanelThreads, sm, c);
      if (act < 1) continue;
      const int waves = (std::max(batch, 1) + act - 1) / act;
      if (!found || waves < best_waves) {  // candidates come wider first, then smaller clusters
        found = true;
        best_waves = waves;
        nb = w;
        cl = c;
      }
    }
  }
  return found;
}

}  // namespace

namespace {
// Answers of the occupancy queries below, by device and question: a solve asks two of them each
// call (10 queries or so of the driver), and a lane of its own thread asks again.
using PlanKey = std::array<int, 5>;  // device, form, order, width wanted (-1: resident batch), batch
struct PanelPlan {
  bool ok = false;
  int nb = 0, cl = 0, resident = 0;
};
template <typename F> PanelPlan remembered_plan(PlanKey key, F&& find) {
  static std::mutex mu;
  static std::map<PlanKey, PanelPlan> known;
  int dev = 0;
  cudaGetDevice(&dev);
  key[0] = dev;
  {
    std::lock_guard<std::mutex> lock(mu);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
  }
  const PanelPlan p = find();
  if (!p.ok) return p;  // a query may fail for want of memory: asked again next time
  std::lock_guard<std::mutex> lock(mu);
  if (known.size() >= 4096) known.clear();
  return known[key] = p;
}
}  // namespace

bool lu_cluster_plan(Precision prec, int n, int want_nb, int batch, int* nb, int* cl) {
  const PanelPlan p = remembered_plan({0, (int)prec, n, want_nb, batch}, [&] {
    PanelPlan q;
    q.ok = prec == Precision::Mixed ? choose_panel<float>(n, want_nb, batch, q.nb, q.cl)
                                    : choose_panel<double>(n, want_nb, batch, q.nb, q.cl);
    return q;
  });
  *nb = p.nb;
  *cl = p.cl;
  return p.ok;
}

// Matrices whose cluster panels are resident at once (one wave) for an n x n
// factorisation with the panel plan of a large batch: a batch beyond this
// runs every panel in two waves.
namespace {
bool resident_batch(Precision prec, int n, int* resident) {
  int nb = 0, cl = 0;
  *resident = 64;
  if (!lu_cluster_plan(prec, n, 0, 64, &nb, &cl)) return false;
  const int chunk = (n + cl - 1) / cl;
  int act = 0;
  if (prec == Precision::Mixed && nb == 32 && chunk <= kRegPanelThreads)
    act = cl > 1 ? active_clusters(lu_panel_reg_kernel<true>, kRegPanelThreads,
                                   (size_t)32 * kRegPanelThreads * sizeof(float2), cl)
                 : active_clusters(lu_panel_reg_kernel<false>, kRegPanelThreads,
                                   (size_t)32 * kRegPanelThreads * sizeof(float2), cl);
  else if (prec == Precision::Mixed)
    act = nb == 64 ? active_clusters(lu_panel_cluster_kernel<float, 64>, kPanelThreads, panel_smem<float, 64>(chunk), cl)
                   : active_clusters(lu_panel_cluster_kernel<float, 32>, kPanelThreads, panel_smem<float, 32>(chunk), cl);
  else if (nb == 32 && chunk <= kReg64Threads)
    act = active_clusters(lu_panel_reg64_kernel, kReg64Threads, kReg64Smem, cl);
  else
    act = nb == 64 ? active_clusters(lu_panel_cluster_kernel<double, 64>, kPanelThreads, panel_smem<double, 64>(chunk), cl)
                   : active_clusters(lu_panel_cluster_kernel<double, 32>, kPanelThreads, panel_smem<double, 32>(chunk), cl);
  *resident = std::max(1, act);
  return true;
}
}  // namespace

int lu_resident_batch(Precision prec, int n) {
  return remembered_plan({0, (int)prec, n, -1, 64}, [&] {
           PanelPlan q;
           q.ok = resident_batch(prec, n, &q.resident);
           return q;
         }).resident;
}

cudaError_t lu_panel_cluster(Precision prec, void* A, long long lda, long long strideA, int n, int k, int kb, int nb,
                             int cl, int batch, int* ipiv, int* info, cudaStream_t stream, int* rowmap, int polls) {
  const int m = n - k;
  const int chunk = (m + cl - 1) / cl;
  void* args[] = {&A, &lda, &strideA, &n, &k, &kb, (void*)&chunk, &ipiv, &info, &rowmap, &polls};  // polls: register panels
  dim3 grid(cl, batch);
  if (prec == Precision::Mixed && nb == 32 && chunk <= kRegPanelThreads && kb == 32) {
    const size_t sm = (size_t)32 * kRegPanelThreads * sizeof(float2);
    if (cl == 1) {
      ensure_smem_limit((const void*)lu_panel_reg_kernel<false>, sm);
      return launch_cluster(lu_panel_reg_kernel<false>, grid, kRegPanelThreads, sm, cl, stream, args, true);
    }
    ensure_smem_limit((const void*)lu_panel_reg_kernel<true>, sm);
    cudaFuncSetAttribute(lu_panel_reg_kernel<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return launch_cluster(lu_panel_reg_kernel<true>, grid, kRegPanelThreads, sm, cl, stream, args, true);
  }
  if (prec == Precision::Mixed) {
    if (nb == 64) {
      const size_t sm = panel_smem<float, 64>(chunk);
      ensure_smem_limit((const void*)lu_panel_cluster_kernel<float, 64>, sm);
      cudaFuncSetAttribute(lu_panel_cluster_kernel<float, 64>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      return launch_cluster(lu_panel_cluster_kernel<float, 64>, grid, kPanelThreads, sm, cl, stream, args);
    }
    const size_t sm = panel_smem<float, 32>(chunk);
    ensure_smem_limit((const void*)lu_panel_cluster_kernel<float, 32>, sm);
    cudaFuncSetAttribute(lu_panel_cluster_kernel<float, 32>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return launch_cluster(lu_panel_cluster_kernel<float, 32>, grid, kPanelThreads, sm, cl, stream, args);
  }
  if (nb == 32 && kb == 32 && chunk <= kReg64Threads) {
    ensure_smem_limit((const void*)lu_panel_reg64_kernel, kReg64Smem);
    cudaFuncSetAttribute(lu_panel_reg64_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return launch_cluster(lu_panel_reg64_kernel, grid, kReg64Threads, kReg64Smem, cl, stream, args);
  }
  if (nb == 64) {
    const size_t sm = panel_smem<double, 64>(chunk);
    ensure_smem_limit((const void*)lu_panel_cluster_kernel<double, 64>, sm);
    cudaFuncSetAttribute(lu_panel_cluster_kernel<double, 64>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return launch_cluster(lu_panel_cluster_kernel<double, 64>, grid, kPanelThreads, sm, cl, stream, args);
  }
  const size_t sm = panel_smem<double, 32>(chunk);
  ensure_smem_limit((const void*)lu_panel_cluster_kernel<double, 32>, sm);
  cudaFuncSetAttribute(lu_panel_cluster_kernel<double, 32>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return launch_cluster(lu_panel_cluster_kernel<double, 32>, grid, kPanelThreads, sm, cl, stream, args);
}

cudaError_t lu_swap_rows_batched(Precision prec, void* A, long long lda, long long strideA, int n, int k, int kb,
                                 int batch, const int* rowmap, int* perm, cudaStream_t stream) {
  const int warps = n - kb + (perm ? 1 : 0);
  if (warps <= 0) return cudaSuccess;
  dim3 g((unsigned)((warps + 7) / 8), batch);
  if (prec == Precision::Mixed)
    lu_swap_rows_kernel<float2><<<g, 256, 0, stream>>>((float2*)A, lda, strideA, n, k, kb, rowmap, perm);
  else
    lu_swap_rows_kernel<double2><<<g, 256, 0, stream>>>((double2*)A, lda, strideA, n, k, kb, rowmap, perm);
  return cudaGetLastError();
}

cudaError_t lu_perm_batched(const int* ipiv, int n, int batch, int* perm, cudaStream_t stream) {
  const size_t sm = (size_t)n * sizeof(int);
  if (sm > 48 * 1024) ensure_smem_limit((const void*)lu_perm_kernel, sm);
  lu_perm_kernel<<<batch, 256, sm, stream>>>(ipiv, n, perm);
  return cudaGetLastError();
}

cudaError_t lu_solve_cluster_batched(Precision prec, const void* LU, long long lda, int n, int batch, const int* perm,
                                     void* B, long long ldb, int nrhs, cudaStream_t stream) {
  const long long strideA = lda * (long long)n;
  const size_t esz = prec == Precision::Mixed ? sizeof(float2) : sizeof(double2);
  // rows per CTA: a multiple of 32 so that each 32-row block has one owner
  int cl = 8;
  int chunk = ((n + cl - 1) / cl + 31) / 32 * 32;
  const size_t sm = (size_t)(chunk + 64) * esz;
  dim3 grid(cl, batch * nrhs);
  if (prec == Precision::Mixed) {
    ensure_smem_limit((const void*)lu_solve_cluster_kernel<float>, sm);
    void* args[] = {&LU, &lda, (void*)&strideA, &n, &perm, &B, &ldb, &nrhs, &chunk};
    return launch_cluster(lu_solve_cluster_kernel<float>, grid, kSolveThreads, sm, cl, stream, args);
  }
  ensure_smem_limit((const void*)lu_solve_cluster_kernel<double>, sm);
  void* args[] = {&LU, &lda, (void*)&strideA, &n, &perm, &B, &ldb, &nrhs, &chunk};
  return launch_cluster(lu_solve_cluster_kernel<double>, grid, kSolveThreads, sm, cl, stream, args);
}

}  // namespace bem
