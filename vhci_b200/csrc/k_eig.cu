// Lowest eigenpairs of a small dense symmetric matrix (the projected matrix of the Lanczos solver,
// 100 to 640 rows, once per cycle; the first dense heat-bath steps), the role of the dense
// eigensolvers behind Spectra and Eigen in the reference (Ham.cpp:347-379).
//
//   1. k_tridiag: Householder tridiagonalisation in one cluster of thread blocks that hold the whole
//      matrix in their shared memory (rows dealt cyclically), one cluster barrier a column; beyond
//      640 rows k_tridiag_grid, the same over all SMs; the last 128 columns, and matrices that have no
//      more, by k_tridiag_block, one block with the matrix in its registers;
//   2. k_tri_vectors: one warp per wanted eigenvalue: Sturm counts at 32 points a round, then the
//      vector from the twisted factorisation of T - lambda I;
//   3. two Newton-Schulz steps Z <- Z (3 I - Z^T Z) / 2 take out the mixing of close eigenvalues
//      (k_eig_gram, k_eig_mul, FP64 tensor cores), with the deviation from orthonormality before each;
//   4. k_back: the reflectors applied to the vectors, one warp per vector.
//
// All steps at 192, 352 and 640 rows (half of the vectors wanted) took 0.66, 1.4 and 3.7 ms, against
// 1.9, 3.5 and 7 ms for syevd with its host steps, when step 1 was k_tridiag alone (0.42, 0.99 and
// 2.9 ms); with the last 128 columns in one block step 1 takes 0.30 ms at 192 rows and 0.82 at 352.
//
// Vectors of eigenvalues closer than about 1e-12 of the norm come out too far from orthogonal for
// step 3; the deviations tell, and the caller takes the library's solver instead.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdint>
#include <mutex>

#include "chain.cuh"
#include "ops.h"

namespace cg = cooperative_groups;

namespace vhci {

namespace {

constexpr int kTriThreads = 256, kTriWarps = kTriThreads / 32;
constexpr int kTriRows = 8;   // rows a warp holds at most
constexpr int kVecWarps = 4;
constexpr int kTriTail = 128;       // rows of k_tridiag_block
constexpr int kBlockThreads = 256;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The same by the tensor pipe (the order of the lanes is another): 126 cycles against 187 alone on an SM,
// 155 against 189 with eight warps.
__device__ __forceinline__ double warp_sum_mma(double v) {
  double s0 = 0.0, s1 = 0.0, z = 0.0;
  // lane 4 m + k gives element (m, k); times ones: row m's sum, in lanes 4 m .. 4 m + 3
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(s0), "+d"(z) : "d"(v), "d"(1.0));
  const int k = threadIdx.x & 3;
  const double lo = __shfl_sync(0xffffffffu, s0, 4 * k), hi = __shfl_sync(0xffffffffu, s0, 4 * k + 16);
  s0 = s1 = 0.0;
  double z0 = 0.0, z1 = 0.0;
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(s0), "+d"(z0) : "d"(1.0), "d"(lo));
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(s1), "+d"(z1) : "d"(1.0), "d"(hi));
  return s0 + s1;
}

// Sums of N values (a power of two) over the warp, halving the values a lane carries at each step: lane l
// returns the sum of value l N / 32.
template <int N>
__device__ __forceinline__ double warp_sums(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int h = N / 2; h > 0; o >>= 1, h >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int q = 0; q < N / 2; ++q)
      if (q < h) {
        const double give = up ? v[q] : v[q + h], keep = up ? v[q + h] : v[q];
        v[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
  }
  double s = v[0];
#pragma unroll
  for (int x = 16 / N; x > 0; x >>= 1) s += __shfl_xor_sync(0xffffffffu, s, x);
  return s;
}

// Dynamic shared memory: the block's rows (m values each), p and the next row as they arrive (two
// buffers each), v at the block's own rows (two buffers).
__host__ __device__ constexpr size_t tri_smem(int m, int blocks) {
  const size_t rows = (size_t)((m + blocks - 1) / blocks);
  return (rows * m + 4 * (size_t)m + 2 * rows) * sizeof(double);
}

// A = H_0 .. H_{m-3} (tridiagonal d, e) H_{m-3} .. H_0 with H_k = I - tau_k v_k v_k^T, v_k (zero up to
// k, one at k + 1) in row k of V.  T holds the upper triangle of A, column-major.  m <= 32 NR.
//
// Row l C + r of the matrix is kept by block r of the cluster, in its warp l % kTriWarps.  Column k
// takes one cluster barrier: every warp of every block holds v_{k-1} in registers (columns lane + 32 q)
// and finds p_{k-1} = tau A v_{k-1} and row k, as it was before the update with them, in its block's
// shared memory; it forms the updated row k, the reflector v_k and tau_k from it by itself, then in
// one pass over its own rows applies the update A - v p^T - (p + K v) v^T, K = - tau v^T p, and
// multiplies by v_k, and hands p_k and (the keeper of that row) row k + 1 to all blocks.  Bound by
// latency: the barrier, three warp sums, a square root and a division a column.  Measured at 192, 352
// and 640 rows, to the last column: 0.42, 0.99 and 2.9 ms (now it stops 128 columns before: 0.15 and
// 0.67 ms at 192 and 352); with two barriers, one of which waits for one block to form v and hand it
// round, 0.72, 1.8 and 4.9 ms; the tridiagonalisation of cuSOLVER's syevd takes 1.0 ms at 192 and 2.5
// at 352.  The barriers wait only for blocks of the same cluster, which run together.
template <int NR>
__global__ void __launch_bounds__(kTriThreads) k_tridiag(const double* __restrict__ T, int ldt, int m,
                                                         double* __restrict__ d, double* __restrict__ e,
                                                         double* __restrict__ tau,
                                                         double* __restrict__ V, double* rowx,
                                                         double* __restrict__ tail) {
  constexpr bool kRowGlobal = NR > 8;
  extern __shared__ double sm[];
  cg::cluster_group cl = cg::this_cluster();
  const int C = (int)cl.num_blocks(), r = (int)cl.block_rank();
  const int sh = 31 - __clz(C), lm = C - 1;  // C is a power of two
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int R = (m + C - 1) / C;
  double* A = sm;                     // local row l is row l C + r
  double* sp = A + (size_t)R * m;     // [2][m] p
  double* srow = sp + 2 * m;          // [2][m] the next row
  double* svr = srow + 2 * m;         // [2][R] v at the local rows
  const int rows = r < m ? (m - r + C - 1) / C : 0;
  for (int l = wid; l < rows; l += kTriWarps) {
    const int i = l * C + r;
    for (int j = lane; j < m; j += 32)
      A[(size_t)l * m + j] = i <= j ? T[i + (int64_t)j * ldt] : T[j + (int64_t)i * ldt];
  }
  for (int j = tid; j < m; j += kTriThreads) {
    sp[j] = 0.0;
    const double y = T[(int64_t)j * ldt];  // row 0
    srow[j] = y;
    if (kRowGlobal && r == 0) rowx[j] = y;
  }
  for (int l = tid; l < 2 * R; l += kTriThreads) svr[l] = 0.0;
  double v[NR];  // v_{k-1}
#pragma unroll
  for (int q = 0; q < NR; ++q) v[q] = 0.0;
  double t = 0.0;  // tau_{k-1}
  cl.sync();
  const int k0 = m - kTriTail;
  for (int k = 0; k < k0; ++k) {
    const int par = k & 1, q0 = (k + 1) >> 5;  // chunks before q0 are done
    const double* p_in = sp + par * m;
    double p[NR], x[NR], s = 0.0, s1 = 0.0;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const int j = lane + 32 * q;
      const bool in = j >= k && j < m;
      p[q] = in ? p_in[j] : 0.0;
      x[q] = !in ? 0.0 : kRowGlobal ? __ldcg(rowx + par * m + j) : srow[par * m + j];
    }
#pragma unroll
    for (int q = 0; q < NR; ++q)
      if (q & 1) s1 = fma(v[q], p[q], s1); else s = fma(v[q], p[q], s);
    const double K = -t * warp_sum_mma(s + s1);
    {  // row k, updated
      const double vk = k > 0 ? 1.0 : 0.0, ck = fma(K, vk, p_in[k]);
      s = s1 = 0.0;
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const int j = lane + 32 * q;
        x[q] -= fma(vk, p[q], ck * v[q]);
        const double y = j > k + 1 ? x[q] : 0.0;
        if (q & 1) s1 = fma(y, y, s1); else s = fma(y, y, s);
      }
    }
    const double ss = warp_sum_mma(s + s1);
    double alpha = 0.0;
#pragma unroll
    for (int q = 0; q < NR; ++q)
      if (q == q0) alpha = x[q];
    alpha = __shfl_sync(0xffffffffu, alpha, (k + 1) & 31);
    double beta = alpha, inv = 0.0, tn = 0.0;
    if (ss > 0.0 && k + 2 < m) {
      beta = -copysign(sqrt(fma(alpha, alpha, ss)), alpha);
      const double g = 1.0 / (beta * (alpha - beta));  // both quotients from one division
      inv = beta * g;
      tn = (beta - alpha) * ((alpha - beta) * g);
    }
    const bool keeper = r == (k & lm) && wid == 0;
    double vn[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const int j = lane + 32 * q;
      vn[q] = j > k + 1 ? x[q] * inv : (j == k + 1 ? 1.0 : 0.0);
      if (keeper) {
        if (j == k) d[k] = x[q];
        if (j > k && j < m) V[(int64_t)k * m + j] = vn[q];
      }
      if (wid == 0 && j < m && (j & lm) == r) svr[par * R + (j >> sh)] = vn[q];
    }
    if (keeper && lane == 0) {
      e[k] = beta;
      tau[k] = tn;
    }
    // own rows below k: update with v, p; multiply by the new reflector
    const double* vr = svr + (par ^ 1) * R;
    const int lr = (k + 1) >> sh;
    const bool has_next = r == ((k + 1) & lm);  // this block keeps row k + 1
    double sum[kTriRows];
    auto pass = [&](int l, bool out) -> double {
      const int i = (l << sh) + r;
      const double vi = vr[l], ci = fma(K, vi, p_in[i]);
      double* a = A + (size_t)l * m;
      double y[NR], u = 0.0, u1 = 0.0;
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const int j = lane + 32 * q;
        y[q] = q >= q0 && j < m ? a[j] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < NR; ++q) y[q] -= fma(vi, p[q], ci * v[q]);
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const int j = lane + 32 * q;
        if (q >= q0 && j < m) a[j] = y[q];
        if (kRowGlobal && out && q >= q0 && j < m) __stcg(rowx + (par ^ 1) * m + j, y[q]);
        if (q & 1) u1 = fma(y[q], vn[q], u1); else u = fma(y[q], vn[q], u);
      }
      return u + u1;
    };
    // the keeper of row k + 1 updates it first; it goes to all blocks through their shared memory by
    // the whole block, or for long rows (320 stores a lane otherwise) through L2
    double first = 0.0;
    if (has_next) {
      if (wid == lr % kTriWarps) first = pass(lr, true);
      if (!kRowGlobal) {
        __syncthreads();
        for (int j = k + 1 + tid; j < m; j += kTriThreads) {
          const double y = A[(size_t)lr * m + j];
          for (int c = 0; c < C; ++c) cl.map_shared_rank(srow, c)[(par ^ 1) * m + j] = y;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kTriRows; ++q) {
      const int l = wid + q * kTriWarps;
      sum[q] = 0.0;
      if (l < rows && (l << sh) + r > k) sum[q] = has_next && l == lr ? first : pass(l, false);
    }
    {
      const double pi = tn * warp_sums<kTriRows>(sum);
      const int l = wid + (lane / 4) * kTriWarps, i = (l << sh) + r;
      if (l < rows && i > k)
        for (int c = lane & 3; c < C; c += 4) cl.map_shared_rank(sp, c)[(par ^ 1) * m + i] = pi;
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) v[q] = vn[q];
    t = tn;
    cl.sync();  // p and the next row have arrived
  }
  // the rest of the matrix, with its last update, for k_tridiag_block
  const double* p_in = sp + (k0 & 1) * m;
  const double* vr = svr + ((k0 & 1) ^ 1) * R;
  double p[NR], s = 0.0;
#pragma unroll
  for (int q = 0; q < NR; ++q) {
    const int j = lane + 32 * q;
    p[q] = j >= k0 && j < m ? p_in[j] : 0.0;
    s = fma(v[q], p[q], s);
  }
  const double K = -t * warp_sum(s);
  for (int l = wid; l < rows; l += kTriWarps) {
    const int i = (l << sh) + r;
    if (i < k0) continue;
    const double vi = vr[l], ci = fma(K, vi, p_in[i]);
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      const int j = lane + 32 * q;
      if (j >= k0 && j < m)
        tail[(i - k0) * kTriTail + j - k0] = A[(size_t)l * m + j] - fma(vi, p[q], ci * v[q]);
    }
  }
}

// The same for matrices beyond one cluster's shared memory (m <= kSmallEigMax), over the whole GPU: row
// l G + r of the matrix is kept by block r of G in its shared memory, and a thread works on columns
// tid + kGridThreads c of all the block's rows, so that v, p and the row being reduced stay in its
// registers.  p and the next row go through L2, and the blocks meet once a column: block 0 .. G - 1
// each count up *ctr, and wait for all with a limit, after which *err is set and the kernel gives up
// (launched cooperatively, so that all blocks run together).  Bound by latency: the meeting and the
// exchange (2 us), two block sums, a square root and a division a column.  Measured at 672, 1,225 and
// 1,500 rows, to the last column, 3.0, 6.1 and 7.6 ms (one cluster at 640: 2.9; at 672 now 2.52, 128
// columns short of the last); the whole solve 4.0, 7.8 and 9.7 ms, where
// cuSOLVER's syevd takes 7.8, 15.6 and 19.6.
constexpr int kGridThreads = 512, kGridWarps = kGridThreads / 32;
constexpr int kGridCols = 4;    // columns a thread: m <= 2048
constexpr int kGridRows = 16;   // rows a block
__device__ __forceinline__ double grid_block_sum(double v, double (&red)[2][kGridWarps], int& buf) {
  const int lane = threadIdx.x & 31;
  v = warp_sum(v);
  if (lane == 0) red[buf][threadIdx.x >> 5] = v;
  __syncthreads();
  double t = red[buf][lane % kGridWarps];
#pragma unroll
  for (int o = kGridWarps / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  buf ^= 1;
  return t;
}

__global__ void __launch_bounds__(kGridThreads, 1) k_tridiag_grid(
    const double* __restrict__ T, int ldt, int m, double* __restrict__ d, double* __restrict__ e,
    double* __restrict__ tau, double* __restrict__ V, double* xch, unsigned long long* ctr,
    unsigned long long* err, double* __restrict__ tail, int max_polls) {
  extern __shared__ double sm[];
  __shared__ double red[2][kGridWarps], s_v[kGridRows], s_p[kGridRows], s_x[2];
  __shared__ double s_part[kGridWarps][kGridRows];
  __shared__ int s_stop;
  const int G = gridDim.x, r = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double* A = sm;  // local row l is row l G + r
  const int rows = r < m ? (m - r + G - 1) / G : 0;
  for (int l = wid; l < rows; l += kGridWarps) {
    const int i = l * G + r;
    for (int j = lane; j < m; j += 32)
      A[(size_t)l * m + j] = i <= j ? T[i + (int64_t)j * ldt] : T[j + (int64_t)i * ldt];
  }
  int own[kGridCols];  // local row with this column's index, or -1
  double v[kGridCols], p[kGridCols], x[kGridCols];
#pragma unroll
  for (int c = 0; c < kGridCols; ++c) {
    const int j = tid + kGridThreads * c;
    own[c] = j < m && j % G == r ? j / G : -1;
    v[c] = p[c] = 0.0;
    x[c] = j < m ? T[(int64_t)j * ldt] : 0.0;  // row 0
  }
  if (tid < kGridRows) s_v[tid] = s_p[tid] = 0.0;
  if (tid == 0) s_stop = 0;
  __syncthreads();
  double t = 0.0;
  int buf = 0;
  const int k0 = m - kTriTail;
  for (int k = 0; k <= k0; ++k) {
    const int par = k & 1;
    if (k > 0) {
      if (tid == 0) {  // all blocks have handed on p and row k
        const unsigned long long want = (unsigned long long)k * G;
        unsigned long long seen = 0;
        int polls = 0;
        do {
          asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(ctr) : "memory");
        } while (seen < want && ++polls < max_polls);
        if (seen < want) {
          s_stop = 1;
          *err = 1;
        }
        __threadfence();
      }
      __syncthreads();
      if (s_stop) return;
#pragma unroll
      for (int c = 0; c < kGridCols; ++c) {
        const int j = tid + kGridThreads * c;
        const bool in = j >= k && j < m;
        p[c] = in ? __ldcg(xch + (size_t)par * 2 * m + j) : 0.0;
        x[c] = in ? __ldcg(xch + (size_t)par * 2 * m + m + j) : 0.0;
        if (own[c] >= 0) s_p[own[c]] = p[c];
        if (j == k) s_x[0] = p[c];
      }
    }
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < kGridCols; ++c) s = fma(v[c], p[c], s);
    const double K = -t * grid_block_sum(s, red, buf);
    if (k == k0) {
      t = K;
      break;
    }
    const double vk = k > 0 ? 1.0 : 0.0, ck = k > 0 ? s_x[0] + K : 0.0;
    s = 0.0;
#pragma unroll
    for (int c = 0; c < kGridCols; ++c) {
      const int j = tid + kGridThreads * c;
      x[c] -= fma(vk, p[c], ck * v[c]);
      if (j > k + 1) s = fma(x[c], x[c], s);
      if (j == k + 1) s_x[1] = x[c];
      if (j == k && r == 0) d[k] = x[c];
    }
    const double ss = grid_block_sum(s, red, buf), alpha = s_x[1];
    double beta = alpha, inv = 0.0, tn = 0.0;
    if (ss > 0.0 && k + 2 < m) {
      beta = -copysign(sqrt(fma(alpha, alpha, ss)), alpha);
      const double g = 1.0 / (beta * (alpha - beta));
      inv = beta * g;
      tn = (beta - alpha) * ((alpha - beta) * g);
    }
    if (r == 0 && tid == 0) {
      e[k] = beta;
      tau[k] = tn;
    }
    double vi[kGridRows], sum[kGridRows];
#pragma unroll
    for (int l = 0; l < kGridRows; ++l) {
      vi[l] = s_v[l];
      sum[l] = 0.0;
    }
    const int lr = (k + 1) / G;
    const bool has_next = r == (k + 1) % G;
#pragma unroll
    for (int c = 0; c < kGridCols; ++c) {
      const int j = tid + kGridThreads * c;
      const double y = j > k + 1 ? x[c] * inv : (j == k + 1 ? 1.0 : 0.0);
      if (j > k && j < m) {
        if (r == k % G) V[(int64_t)k * m + j] = y;
#pragma unroll
        for (int l = 0; l < kGridRows; ++l) {
          if (l < rows && l * G + r > k) {
            const double a = A[(size_t)l * m + j] - fma(vi[l], p[c], fma(K, vi[l], s_p[l]) * v[c]);
            A[(size_t)l * m + j] = a;
            sum[l] = fma(a, y, sum[l]);
            if (has_next && l == lr) __stcg(xch + (size_t)(par ^ 1) * 2 * m + m + j, a);
          }
        }
      }
      x[c] = y;
    }
    const double wsum = warp_sums<kGridRows>(sum);
    if ((lane & 1) == 0) s_part[wid][lane >> 1] = wsum;
    __syncthreads();  // also: every thread has read s_v and s_p
    {
      double q = s_part[lane % kGridWarps][wid];  // row wid over the warps
#pragma unroll
      for (int o = kGridWarps / 2; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
      const int i = wid * G + r;
      if (lane == 0 && wid < rows && i > k) __stcg(xch + (size_t)(par ^ 1) * 2 * m + i, tn * q);
    }
#pragma unroll
    for (int c = 0; c < kGridCols; ++c) {
      v[c] = x[c];
      if (own[c] >= 0) s_v[own[c]] = x[c];
    }
    t = tn;
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      atomicAdd(ctr, 1ull);
    }
  }
  // the rest of the matrix, with its last update (t: K), for k_tridiag_block
#pragma unroll
  for (int c = 0; c < kGridCols; ++c) {
    const int j = tid + kGridThreads * c;
    if (j < k0 || j >= m) continue;
    for (int l = 0; l < rows; ++l)
      if (l * G + r >= k0)
        tail[(l * G + r - k0) * kTriTail + j - k0] =
            A[(size_t)l * m + j] - fma(s_v[l], p[c], fma(t, s_v[l], s_p[l]) * v[c]);
  }
}

// A warp's share of a column in k_tridiag_block: its rows from 32 C0 on, in the columns from 32 C0 on,
// updated (A - v w^T - w v^T, w = p + K / 2 v, K2 = K / 2) and multiplied by the new reflector vn; row k + 1 is put out.
template <int C0>
__device__ __forceinline__ void block_pass(double (&a)[16][4], double (&sum)[16], const double (&w)[4],
                                           const double (&v)[4], const double (&vn)[4], double K2,
                                           const double* sv, const double* sp, double* srow, int k, int wid,
                                           int lane) {
#pragma unroll
  for (int q = 0; q < 16; ++q) sum[q] = 0.0;
#pragma unroll
  for (int q = 4 * C0; q < 16; ++q) {
    const int i = 8 * q + wid;
    const double vi = i > k ? -sv[i] : 0.0, wi = i > k ? fma(K2, vi, -sp[i]) : 0.0;  // -v, -w
#pragma unroll
    for (int c = C0; c < 4; ++c) a[q][c] = fma(wi, v[c], fma(vi, w[c], a[q][c]));
#pragma unroll
    for (int c = C0; c < 4; ++c) sum[q] = fma(a[q][c], vn[c], sum[q]);
  }
  if (wid == ((k + 1) & 7))
#pragma unroll
    for (int q = 4 * C0; q < 16; ++q)
      if (8 * q + wid == k + 1)
#pragma unroll
        for (int c = C0; c < 4; ++c) srow[lane + 32 * c] = a[q][c];
}

// The same for n <= 128 rows, in one block that holds the matrix in registers: warp w keeps the rows
// 8 q + w, a lane their columns lane + 32 c; p, v and the next row go through shared memory, and the
// block meets once a column.  T holds the upper triangle, column-major; V's rows lie ldv apart.  Bound by
// latency (two warp sums, a square root and a division, the sums of the rows), and at its first columns by
// the FP64 rate of one SM: 128 rows take 155 us, 1.2 us a column (16 warps with the finished rows left out
// by a branch each: 250).  128 rows because half as many again would not fit the registers; it also ends
// the larger matrices, where a column costs a meeting of the cluster (2.3 us at 192 rows) or the grid.
__global__ void __launch_bounds__(kBlockThreads, 1) k_tridiag_block(const double* T, int ldt, int n,
                                                                    double* __restrict__ d,
                                                                    double* __restrict__ e,
                                                                    double* __restrict__ tau,
                                                                    double* __restrict__ V, int ldv) {
  constexpr int W = kBlockThreads / 32, RQ = kTriTail / W, NC = kTriTail / 32;
  static_assert(W == 8 && RQ == 16 && NC == 4, "block_pass is written for these");
  chain_wait();
  __shared__ double sp[2][kTriTail], srow[2][kTriTail], sv[2][kTriTail];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double a[RQ][NC];
#pragma unroll
  for (int q = 0; q < RQ; ++q)
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int i = W * q + wid, j = lane + 32 * c;
      a[q][c] = i < n && j < n ? (i <= j ? T[i + (int64_t)j * ldt] : T[j + (int64_t)i * ldt]) : 0.0;
    }
  if (threadIdx.x < kTriTail) {
    const int j = threadIdx.x;
    sp[0][j] = sp[1][j] = sv[0][j] = sv[1][j] = srow[1][j] = 0.0;
    srow[0][j] = j < n ? T[(int64_t)j * ldt] : 0.0;  // row 0
  }
  double v[NC], t = 0.0;
#pragma unroll
  for (int c = 0; c < NC; ++c) v[c] = 0.0;
  __syncthreads();
  for (int k = 0; k + 1 < n; ++k) {
    const int par = k & 1, c0 = (k + 1) >> 5;  // columns before chunk c0 are done
    double p[NC], x[NC], w[NC], s = 0.0, s1 = 0.0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = lane + 32 * c;
      p[c] = j >= k ? sp[par][j] : 0.0;
      x[c] = j >= k ? srow[par][j] : 0.0;
      if (c & 1) s1 = fma(v[c], p[c], s1); else s = fma(v[c], p[c], s);
    }
    const double K = -t * warp_sum_mma(s + s1);
    const double vk = k > 0 ? 1.0 : 0.0, ck = fma(K, vk, sp[par][k]);
    const double K2 = 0.5 * K;
    s = s1 = 0.0;
    double alpha = 0.0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {  // row k, updated
      const int j = lane + 32 * c;
      x[c] -= fma(vk, p[c], ck * v[c]);
      const double y = j > k + 1 ? x[c] : 0.0;
      if (c & 1) s1 = fma(y, y, s1); else s = fma(y, y, s);
      w[c] = fma(K2, v[c], p[c]);
      if (c == c0) alpha = x[c];
    }
    alpha = __shfl_sync(0xffffffffu, alpha, (k + 1) & 31);
    const double ss = warp_sum_mma(s + s1);
    double beta = alpha, inv = 0.0, tn = 0.0;
    if (ss > 0.0 && k + 2 < n) {
      beta = -copysign(sqrt(fma(alpha, alpha, ss)), alpha);
      const double g = 1.0 / (beta * (alpha - beta));
      inv = beta * g;
      tn = (beta - alpha) * ((alpha - beta) * g);
    }
    double vn[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int j = lane + 32 * c;
      vn[c] = j > k + 1 ? x[c] * inv : (j == k + 1 ? 1.0 : 0.0);
    }
    if (wid == (k & (W - 1))) {
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const int j = lane + 32 * c;
        sv[par][j] = vn[c];
        if (j == k) d[k] = x[c];
        if (j > k && j < n) V[(int64_t)k * ldv + j] = vn[c];
      }
      if (lane == 0) {
        e[k] = beta;
        tau[k] = tn;
      }
    }
    double sum[RQ];
    switch (c0) {  // finished rows and columns are left out 32 at a time, without a branch a row
      case 0: block_pass<0>(a, sum, w, v, vn, K2, sv[par ^ 1], sp[par], srow[par ^ 1], k, wid, lane); break;
      case 1: block_pass<1>(a, sum, w, v, vn, K2, sv[par ^ 1], sp[par], srow[par ^ 1], k, wid, lane); break;
      case 2: block_pass<2>(a, sum, w, v, vn, K2, sv[par ^ 1], sp[par], srow[par ^ 1], k, wid, lane); break;
      default: block_pass<3>(a, sum, w, v, vn, K2, sv[par ^ 1], sp[par], srow[par ^ 1], k, wid, lane); break;
    }
    const double pi = tn * warp_sums<RQ>(sum);
    const int i = W * (lane >> 1) + wid;
    if ((lane & 1) == 0 && i > k) sp[par ^ 1][i] = pi;
#pragma unroll
    for (int c = 0; c < NC; ++c) v[c] = vn[c];
    t = tn;
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < RQ; ++q)
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (W * q + wid == n - 1 && lane + 32 * c == n - 1) d[n - 1] = a[q][c];
}

// Eigenvalue j (j < nk; the last warp takes the largest, for its value alone) of the tridiagonal
// matrix, scaled to norm 1, and its vector in column j of Z (leading dimension m).  Bound by the latency of
// the recurrences: 192 rows take 51 us, 672 rows 170 (with one point a lane and the pivots by division
// 130 and 455).  The Sturm count
// uses the three-term recurrence of the characteristic polynomials (one multiply-add of latency a
// step where the quotient form has a division), rescaled every eight steps; squared off-diagonals
// below 1e-34 are raised to that, a change below the rounding of the matrix.
__global__ void __launch_bounds__(32 * kVecWarps) k_tri_vectors(const double* d,
                                                                const double* e, int m,
                                                                int nk, double* __restrict__ theta,
                                                                double* __restrict__ Z) {
  chain_wait();
  extern __shared__ double sm[];
  __shared__ double s_red[kVecWarps];
  double* sd = sm;              // [m]
  double* se = sd + m;          // [m] off-diagonals, zero at the end
  double* se2 = se + m;         // [m] their squares
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  double* P = se2 + m + (size_t)wid * 2 * m;  // forward pivots, then the vector
  double* M = P + m;                          // backward pivots
  const int fs = m / 8 + 1;
  double* F = se2 + m + (size_t)kVecWarps * 2 * m + (size_t)wid * 2 * fs;  // their rescalings, every 8 rows
  // norm: the largest row sum
  double nrm = 0.0;
  for (int i = tid; i < m; i += blockDim.x) {
    const double a = i > 0 ? fabs(e[i - 1]) : 0.0, b = i + 1 < m ? fabs(e[i]) : 0.0;
    nrm = fmax(nrm, a + fabs(d[i]) + b);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
  if (lane == 0) s_red[wid] = nrm;
  __syncthreads();
  nrm = s_red[0];
#pragma unroll
  for (int q = 1; q < kVecWarps; ++q) nrm = fmax(nrm, s_red[q]);
  const double scale = nrm > 0.0 ? 1.0 / nrm : 1.0;
  for (int i = tid; i < m; i += blockDim.x) {
    const double x = i + 1 < m ? e[i] * scale : 0.0;
    sd[i] = d[i] * scale;
    se[i] = x;
    se2[i] = fmax(x * x, 1e-34);
  }
  __syncthreads();
  const int w = blockIdx.x * kVecWarps + wid;
  if (w > nk || (w == nk && nk >= m)) return;
  const int j = w < nk ? w : m - 1;

  // eigenvalue j lies in [lo, hi): counts of the eigenvalues below 64 points inside, two a lane, whose
  // recurrences overlap
  double lo = -1.0000001, hi = 1.0000001;
  for (int round = 0; round < 10; ++round) {
    const double wd = (hi - lo) * (1.0 / 65.0);
    double x[2], p0[2], p1[2];
    int below[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      x[h] = lo + wd * (2 * lane + h + 1);
      p0[h] = 1.0;
      p1[h] = sd[0] - x[h];
      below[h] = (unsigned)__double2hiint(p1[h]) >> 31;  // sign changes, by the sign bits
    }
    auto step = [&](double di, double e2) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double p2 = fma(di - x[h], p1[h], -e2 * p0[h]);
        below[h] += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1[h])) >> 31;
        p0[h] = p1[h];
        p1[h] = p2;
      }
    };
    auto rescale = [&] {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double big = fmax(fabs(p0[h]), fabs(p1[h]));
        const double f = big > 1e100 ? 1e-100 : (big < 1e-100 ? 1e100 : 1.0);
        p0[h] *= f;
        p1[h] *= f;
      }
    };
    int i = 1;
    for (; i + 8 <= m; i += 8) {
      double di[8], e2[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        di[q] = sd[i + q];
        e2[q] = se2[i + q - 1];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) step(di[q], e2[q]);
      rescale();
    }
    for (; i < m; ++i) step(sd[i], se2[i - 1]);
    const int n = __popc(__ballot_sync(0xffffffffu, below[0] <= j)) +
                  __popc(__ballot_sync(0xffffffffu, below[1] <= j));  // points up to the eigenvalue
    const double l0 = lo;
    if (n > 0) lo = l0 + wd * n;
    if (n < 64) hi = l0 + wd * (n + 1);
    if (hi - lo <= 1e-17) break;
  }
  const double lam = 0.5 * (lo + hi);
  if (lane == 0) theta[j] = lam * nrm;
  if (w >= nk) return;

  // twisted factorisation of T - lam: forward pivots by lane 0, backward ones by lane 1, at once.  The
  // lanes run the recurrence of the characteristic polynomials too; a pivot is the ratio of two that follow
  // one another, and all lanes take the ratios afterwards (with a division in the recurrence, one lane
  // after the other, 192 rows took 26 us more).
  constexpr double tiny = 1e-17;
  if (lane < 2) {
    double* out = lane ? M : P;
    double* fo = F + lane * fs;
    const int s = lane ? -1 : 1, o = lane ? m - 1 : 0, o2 = lane ? m - 1 : -1;  // row of step i: o + s i
    double p0 = 1.0, p1 = sd[o] - lam;
    if (fabs(p1) < tiny) p1 = copysign(tiny, p1);
    out[o] = p1;
    for (int i = 1; i < m; i += 8) {
      double di[8], e2[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const bool in = i + q < m;
        di[q] = in ? sd[o + s * (i + q)] - lam : 0.0;
        e2[q] = in ? se2[o2 + s * (i + q)] : 0.0;
      }
      const double big = fmax(fabs(p0), fabs(p1));
      const double f = big > 1e100 ? 1e-100 : (big < 1e-100 ? 1e100 : 1.0);
      p0 *= f;
      p1 *= f;
      fo[i >> 3] = f;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        double p2 = fma(di[q], p1, -e2[q] * p0);
        const double least = tiny * fabs(p1);
        if (fabs(p2) < least) p2 = copysign(least, p2);
        if (i + q < m) out[o + s * (i + q)] = p2;
        p0 = p1;
        p1 = p2;
      }
    }
  }
  __syncwarp();
  for (int c = (m - 1) / 32 * 32; c >= 0; c -= 32) {  // forward ones from the end, backward ones from row 0
    const int i = c + lane, jr = m - 1 - i;
    double q = 0.0, r = 0.0;
    if (i < m) {
      const bool f = (i & 7) == 1;
      q = i > 0 ? P[i] / (P[i - 1] * (f ? F[i >> 3] : 1.0)) : P[0];
      r = i > 0 ? M[jr] / (M[jr + 1] * (f ? F[fs + (i >> 3)] : 1.0)) : M[jr];
    }
    __syncwarp();
    if (i < m) {
      P[i] = q;
      M[jr] = r;
    }
    __syncwarp();
  }
  double best = 1e300;
  int twist = 0;
  for (int i = lane; i < m; i += 32) {
    const double g = fabs(P[i] + M[i] - (sd[i] - lam));
    if (g < best) { best = g; twist = i; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int ot = __shfl_xor_sync(0xffffffffu, twist, o);
    if (ob < best || (ob == best && ot < twist)) { best = ob; twist = ot; }
  }
  // ratios of neighbouring components, then their running products away from the twist
  __syncwarp();
  for (int i = lane; i < m; i += 32) {
    const double up = i < twist ? -se[i] / P[i] : 0.0;        // z_i = up z_{i+1}
    const double dn = i > twist ? -se[i - 1] / M[i] : 0.0;    // z_i = dn z_{i-1}
    P[i] = i < twist ? up : (i > twist ? dn : 1.0);
  }
  __syncwarp();
  if (lane < 2) {
    const int s = lane ? 1 : -1, n = lane ? m - 1 - twist : twist;
    double z = 1.0, next = n > 0 ? P[twist + s] : 0.0;
    for (int x = 1; x <= n; ++x) {
      const double y = next;
      next = x < n ? P[twist + s * (x + 1)] : 0.0;
      P[twist + s * x] = z = y * z;
    }
  }
  __syncwarp();
  double s = 0.0;
  for (int i = lane; i < m; i += 32) s = fma(P[i], P[i], s);
  s = 1.0 / sqrt(warp_sum(s));
  for (int i = lane; i < m; i += 32) Z[(int64_t)j * m + i] = P[i] * s;
}

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// One warp per 8 x 32 tile of S = (3 I - Z^T Z) / 2 (nk x nk); *dev: the largest |Z^T Z - I| seen, as
// the bits of a non-negative double.
__global__ void __launch_bounds__(128) k_eig_gram(const double* Z, int m, int nk,
                                                  double* __restrict__ S,
                                                  unsigned long long* __restrict__ dev) {
  chain_wait();
  const int lane = threadIdx.x & 31, w = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int tr = (nk + 7) / 8, tc = (nk + 31) / 32;
  if (w >= tr * tc) return;
  const int a0 = (w / tc) * 8, b0 = (w % tc) * 32;
  const int q = lane >> 2, kl = lane & 3;
  double acc[4][2];
#pragma unroll
  for (int u = 0; u < 4; ++u) acc[u][0] = acc[u][1] = 0.0;
  const double* za = Z + (int64_t)min(a0 + q, nk - 1) * m;
  for (int k0 = 0; k0 < m; k0 += 16) {
    double a[4], b[4][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int k = k0 + 4 * s + kl;
      a[s] = k < m ? za[k] : 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        b[s][u] = k < m ? Z[(int64_t)min(b0 + 8 * u + q, nk - 1) * m + k] : 0.0;
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int u = 0; u < 4; ++u) dmma(acc[u], a[s], b[s][u]);
  }
  double worst = 0.0;
  bool bad = false;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = a0 + q, j = b0 + 8 * u + 2 * kl + h;
      if (i >= nk || j >= nk) continue;
      const double g = acc[u][h] - (i == j ? 1.0 : 0.0);
      bad |= !(fabs(g) < 1e300);
      worst = fmax(worst, fabs(g));
      S[i + (int64_t)j * nk] = (i == j ? 1.0 : 0.0) - 0.5 * g;
    }
  if (bad) worst = 1e300;  // a NaN counts as the largest deviation
  atomicMax(dev, (unsigned long long)__double_as_longlong(worst));
}

// Out (m x nk) = Z S, one warp per 8 x 32 tile.
__global__ void __launch_bounds__(128) k_eig_mul(const double* Z, const double* S,
                                                 int m, int nk, double* __restrict__ Out) {
  chain_wait();
  const int lane = threadIdx.x & 31, w = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int tr = (m + 7) / 8, tc = (nk + 31) / 32;
  if (w >= tr * tc) return;
  const int i0 = (w / tc) * 8, j0 = (w % tc) * 32;
  const int q = lane >> 2, kl = lane & 3;
  double acc[4][2];
#pragma unroll
  for (int u = 0; u < 4; ++u) acc[u][0] = acc[u][1] = 0.0;
  for (int k0 = 0; k0 < nk; k0 += 16) {
    double a[4], b[4][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int k = k0 + 4 * s + kl;
      a[s] = k < nk ? Z[(int64_t)k * m + min(i0 + q, m - 1)] : 0.0;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        b[s][u] = k < nk ? S[(int64_t)min(j0 + 8 * u + q, nk - 1) * nk + k] : 0.0;
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
#pragma unroll
      for (int u = 0; u < 4; ++u) dmma(acc[u], a[s], b[s][u]);
  }
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int i = i0 + q, j = j0 + 8 * u + 2 * kl + h;
      if (i < m && j < nk) Out[i + (int64_t)j * m] = acc[u][h];
    }
}

// Y[:, j] = H_0 .. H_{m-3} Z[:, j], one warp per column with the column in registers (32 NR >= m) and
// the next PF reflectors' loads in flight.
template <int NR, int PF>
__global__ void __launch_bounds__(64) k_back(const double* Z, const double* V,
                                             const double* tau, int m, int nk,
                                             double* __restrict__ Y, int ldy) {
  chain_wait();
  const int lane = threadIdx.x & 31, j = blockIdx.x * 2 + (threadIdx.x >> 5);
  if (j >= nk) return;
  double z[NR], v[PF][NR], t[PF];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int i = lane + 32 * r;
    z[r] = i < m ? Z[(int64_t)j * m + i] : 0.0;
  }
  auto fetch = [&](int k, double (&u)[NR], double& tk) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int i = lane + 32 * r;
      u[r] = (k >= 0 && i > k && i < m) ? V[(int64_t)k * m + i] : 0.0;
    }
    tk = k >= 0 ? tau[k] : 0.0;
  };
#pragma unroll
  for (int f = 0; f < PF; ++f) fetch(m - 3 - f, v[f], t[f]);
  for (int k = m - 3; k >= 0; k -= PF) {
#pragma unroll
    for (int f = 0; f < PF; ++f) {  // a reflector before the first has tau = 0
      double s = 0.0, s1 = 0.0;
#pragma unroll
      for (int r = 0; r < NR; ++r)
        if (r & 1) s1 = fma(v[f][r], z[r], s1); else s = fma(v[f][r], z[r], s);
      s = -t[f] * warp_sum(s + s1);
#pragma unroll
      for (int r = 0; r < NR; ++r) z[r] = fma(s, v[f][r], z[r]);
      fetch(k - f - PF, v[f], t[f]);
    }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int i = lane + 32 * r;
    if (i < m) Y[(int64_t)j * ldy + i] = z[r];
  }
}

// The same with one block of four warps per column (m <= 128 NR).
template <int NR>
__global__ void __launch_bounds__(128) k_back_block(const double* Z, const double* V,
                                                    const double* tau, int m, int nk,
                                                    double* __restrict__ Y, int ldy) {
  chain_wait();
  __shared__ double red[2][4];
  const int tid = threadIdx.x, lane = tid & 31, j = blockIdx.x;
  double z[NR], v[NR], u[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int i = tid + 128 * r;
    z[r] = i < m ? Z[(int64_t)j * m + i] : 0.0;
  }
  auto fetch = [&](int k, double (&w)[NR]) {
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int i = tid + 128 * r;
      w[r] = (k >= 0 && i > k && i < m) ? V[(int64_t)k * m + i] : 0.0;
    }
  };
  fetch(m - 3, v);
  for (int k = m - 3; k >= 0; --k) {
    fetch(k - 1, u);
    const double tk = tau[k];
    double s = 0.0, s1 = 0.0;
#pragma unroll
    for (int r = 0; r < NR; ++r)
      if (r & 1) s1 = fma(v[r], z[r], s1); else s = fma(v[r], z[r], s);
    s = warp_sum(s + s1);
    if (lane == 0) red[k & 1][tid >> 5] = s;
    __syncthreads();
    s = -tk * ((red[k & 1][0] + red[k & 1][1]) + (red[k & 1][2] + red[k & 1][3]));
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      z[r] = fma(s, v[r], z[r]);
      v[r] = u[r];
    }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int i = tid + 128 * r;
    if (i < m) Y[(int64_t)j * ldy + i] = z[r];
  }
}

constexpr size_t vec_smem(int m) {
  return ((size_t)m * (3 + 2 * kVecWarps) + (size_t)(m / 8 + 1) * 2 * kVecWarps) * sizeof(double);
}

// Blocks of the cluster for m rows (its rows must fit the shared memory and kTriRows rounds): 16 (the
// barrier reaches over more of the chip, the pass over the rows is shorter) pay from 256 rows on:
// 0.64 : 0.66 ms there, 0.99 : 1.17 at 352; four are 10 to 20 % slower than eight from 128 on.
int tri_blocks(int m) { return m < 256 ? 8 : 16; }

// Blocks of the grid for m rows: eight rows a block, fewer when the GPU has no more SMs.
int grid_blocks(int m) { return std::min(148, (m + 7) / 8); }
size_t grid_smem(int m) { return (size_t)((m + grid_blocks(m) - 1) / grid_blocks(m)) * m * sizeof(double); }

using TriKernel = void (*)(const double*, int, int, double*, double*, double*, double*, double*, double*);
TriKernel tri_kernel(int m) {
  return m <= 192 ? k_tridiag<6> : m <= 256 ? k_tridiag<8> : m <= 384 ? k_tridiag<12> : k_tridiag<20>;
}

// Polls of k_tridiag_grid's counter before a block gives up (over a second); the tests lower it for their
// thread, to see the wait run out.
constexpr int kGridPolls = 1 << 21;
thread_local int t_grid_polls = kGridPolls;

// Shared-memory and cluster limits of the kernels, set once per device.
constexpr int kMaxDevices = 64;
std::once_flag g_eig_once[kMaxDevices];
bool g_eig_ok[kMaxDevices];

bool eig_attributes() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
  std::call_once(g_eig_once[dev], [dev] {
    bool ok = cudaFuncSetAttribute(k_tri_vectors, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)vec_smem(kSmallEigMax)) == cudaSuccess;
    for (int m : {192, 256, 384, kClusterEigMax}) {
      const TriKernel k = tri_kernel(m);
      ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) == cudaSuccess &&
           cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
    }
    g_eig_ok[dev] = ok && cudaFuncSetAttribute(k_tridiag_grid, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)grid_smem(kSmallEigMax)) == cudaSuccess;
    if (!g_eig_ok[dev]) cudaGetLastError();
  });
  return g_eig_ok[dev];
}

}  // namespace

void small_eig_polls(int polls) { t_grid_polls = polls > 0 ? polls : kGridPolls; }

size_t small_eig_elems(int m, int nk) {
  // d, e, tau; the exchange; V; two vector blocks; S; the last rows
  return 7 * (size_t)m + (size_t)m * m + 2 * (size_t)m * nk + (size_t)nk * nk + kTriTail * kTriTail;
}

bool small_eig(const double* T, int ldt, int m, int nk, double* theta, double* Y, int ldy, double* work,
               unsigned long long* dev, cudaStream_t s) {
  if (m < 1 || m > kSmallEigMax || nk < 1 || nk > m) return false;
  if (!eig_attributes()) return false;
  double* d = work;
  double* e = d + m;
  double* tau = e + m;
  double* rowx = tau + m;
  double* V = rowx + 4 * m;
  double* Za = V + (size_t)m * m;
  double* Zb = Za + (size_t)m * nk;
  double* S = Zb + (size_t)m * nk;
  double* tail = S + (size_t)nk * nk;
  cudaMemsetAsync(dev, 0, kSmallEigDev * sizeof(unsigned long long), s);
  const bool cluster = m <= kClusterEigMax;
  const int k0 = std::max(0, m - kTriTail);  // columns before the last ones
  if (k0 > 0) {
    cudaLaunchConfig_t cfg{};
    cfg.stream = s;
    cudaLaunchAttribute at{};
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t err;
    note_launch();
    if (cluster) {
      const int C = tri_blocks(m);
      cfg.gridDim = dim3(C);
      cfg.blockDim = dim3(kTriThreads);
      cfg.dynamicSmemBytes = tri_smem(m, C);
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = C;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      err = cudaLaunchKernelEx(&cfg, tri_kernel(m), T, ldt, m, d, e, tau, V, rowx, tail);
    } else {
      cfg.gridDim = dim3(grid_blocks(m));
      cfg.blockDim = dim3(kGridThreads);
      cfg.dynamicSmemBytes = grid_smem(m);
      at.id = cudaLaunchAttributeCooperative;
      at.val.cooperative = 1;
      err = cudaLaunchKernelEx(&cfg, k_tridiag_grid, T, ldt, m, d, e, tau, V, rowx, dev + 2, dev + 3, tail, t_grid_polls);
    }
    if (err != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
  }
  note_launch();
  launch_chained(k_tridiag_block, 1, kBlockThreads, 0, s, k0 > 0 ? tail : T, k0 > 0 ? kTriTail : ldt, m - k0,
                 d + k0, e + k0, tau + k0, V + (size_t)k0 * m + k0, m);
  note_launch();
  launch_chained(k_tri_vectors, (nk + 1 + kVecWarps - 1) / kVecWarps, 32 * kVecWarps, vec_smem(m), s, d, e, m, nk,
                                                                                          theta, Za);
  const int tr = (nk + 7) / 8, tc = (nk + 31) / 32, tm = (m + 7) / 8;
  for (int it = 0; it < 2; ++it) {
    note_launch();
    launch_chained(k_eig_gram, (tr * tc + 3) / 4, 128, 0, s, it ? Zb : Za, m, nk, S, dev + it);
    note_launch();
    launch_chained(k_eig_mul, (tm * tc + 3) / 4, 128, 0, s, it ? Zb : Za, S, m, nk, it ? Za : Zb);
  }
  note_launch();
  const int g = (nk + 1) / 2;
  if (m <= 64) launch_chained(k_back<2, 4>, g, 64, 0, s, Za, V, tau, m, nk, Y, ldy);
  else if (m <= 128) launch_chained(k_back<4, 4>, g, 64, 0, s, Za, V, tau, m, nk, Y, ldy);
  else if (m <= 256) launch_chained(k_back<8, 4>, g, 64, 0, s, Za, V, tau, m, nk, Y, ldy);
  else if (m <= 384) launch_chained(k_back<12, 3>, g, 64, 0, s, Za, V, tau, m, nk, Y, ldy);
  else if (cluster) launch_chained(k_back<20, 2>, g, 64, 0, s, Za, V, tau, m, nk, Y, ldy);
  else launch_chained(k_back_block<15>, nk, 128, 0, s, Za, V, tau, m, nk, Y, ldy);
  return true;
}

}  // namespace vhci
