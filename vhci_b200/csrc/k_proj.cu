// FP64 tensor-core projections for the block Lanczos eigensolver (the Gram-Schmidt passes, the
// block orthonormalisation and the Rayleigh-Ritz rotations).  The reference eigensolver (Spectra's
// implicitly restarted Lanczos, Ham.cpp:347-370) does these with Eigen's dense products; here they
// are skinny products over the whole basis, written for B200's FP64 tensor pipe (DMMA,
// mma.sync.m8n8k4.f64).  Both read the tall operand once, straight from global memory into the
// DMMA fragment registers (each lane's fragment element is 8 bytes of a 32-byte row segment, so
// the sectors are fully used), with several k-steps of loads in flight per lane and 32 warps per
// SM; the main loops have no block-wide barriers:
//
//   proj_gram:  C = alpha * A^T B + beta * C   A: n x M, B: n x P (row-major), C: M x P col-major,
//               P <= 16.  A persistent grid splits the n rows over the blocks; each warp keeps
//               the partial products of its 8-row tiles of C in registers; the blocks' partials
//               go to scratch and a second kernel sums them in block order, so the result does not
//               depend on scheduling.
//   proj_rows:  Out = alpha * A S + beta * In    A: n x M row-major, S: M x P col-major,
//               Out: n x P row-major.  Each block holds a 16- or 32-column slab of S in shared memory
//               and its warps stream 8-row tiles of A.  proj_rows_self also forms Out^T Out.
//
// A Lanczos step reads the basis twice (coefficients, update).  Three passes with the first two fused
// over 128-row chunks took 240 + 110 us of projections at 120,011 rows and 512 columns on average,
// 44 us at 24,000 rows and 150 columns; now 140 + 114 and 15 + 13 us.
//
// Fragment layouts of m8n8k4 (row.col): A[m][k] sits in lane 4 m + k, B[k][n] in lane 4 n + k,
// D[m][n] in lane 4 m + n / 2 (element n % 2).
#include <algorithm>
#include <cstdint>
#include <mutex>

#include "ops.h"

namespace vhci {

namespace {

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

constexpr int kThreads = 1024;      // proj_rows: 32 warps, one block per SM
constexpr int kBlocks = 148;
constexpr int kUnroll = 8;          // proj_rows: k-steps of loads issued ahead
constexpr int kGramThreads = 512;   // proj_gram: 16 warps with up to 128 registers each
constexpr int kGramWarps = kGramThreads / 32;
constexpr int kGramTiles = 6;       // 8-row tiles of C per warp: a slab of 16 x 6 x 8 = 768 rows
constexpr int kGramSlab = kGramWarps * kGramTiles * 8;
constexpr int kGramUnroll = 2;

// Partial A^T B over this block's rows for the columns a0 .. a0 + Mc - 1 of A.  The 8-row tiles
// of C are dealt to a group of WG = ceil(tiles / TILES) warps (warp g of a group owns tiles g,
// g + WG, ...); the block's 16 warps form 16 / WG such groups, which take turns over the block's
// rows in steps of 4 UNROLL rows, so a narrow C (few tiles) still keeps every warp streaming.
// When a group would need more than half the warps, all 16 form one group.
// Group r of block x writes its partial to part[x * groups + r] (Mc x P, a-major).
template <int NT, int TILES, int UNROLL, int NWARP>
__global__ void __launch_bounds__(NWARP * 32, 1) k_gram(const double* __restrict__ A, int lda,
                                                    const double* __restrict__ B, int ldb,
                                                    int64_t n, int Mc, int P,
                                                    double* __restrict__ part) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int mt_total = (Mc + 7) / 8;
  int WG = (mt_total + TILES - 1) / TILES;
  if (2 * WG > NWARP) WG = NWARP;  // one group: spread the tiles over all warps
  const int RG = NWARP / WG;
  const int rg = wid / WG, wg = wid - rg * WG;
  if (rg >= RG) return;
  const int64_t per = ((n + gridDim.x - 1) / gridDim.x + 3) & ~int64_t(3);
  const int64_t r0 = (int64_t)blockIdx.x * per, r1 = min(n, r0 + per);
  double acc[TILES][NT][2];
#pragma unroll
  for (int t = 0; t < TILES; ++t)
#pragma unroll
    for (int u = 0; u < NT; ++u) acc[t][u][0] = acc[t][u][1] = 0.0;
  int acol[TILES];
  bool aon[TILES];
#pragma unroll
  for (int t = 0; t < TILES; ++t) {
    acol[t] = 8 * (wg + WG * t) + (lane >> 2);
    aon[t] = (wg + WG * t) < mt_total && acol[t] < Mc;
  }
  const int kl = lane & 3;
  for (int64_t k0 = r0 + 4 * UNROLL * rg; k0 < r1; k0 += 4 * UNROLL * RG) {
    double a[UNROLL][TILES], b[UNROLL][NT];
#pragma unroll
    for (int s = 0; s < UNROLL; ++s) {
      const int64_t i = k0 + 4 * s + kl;
      const bool rin = i < r1;
#pragma unroll
      for (int t = 0; t < TILES; ++t)
        a[s][t] = (rin && aon[t]) ? __ldg(A + i * lda + acol[t]) : 0.0;
#pragma unroll
      for (int u = 0; u < NT; ++u) {
        const int c = 8 * u + (lane >> 2);
        b[s][u] = (rin && c < P) ? __ldg(B + i * ldb + c) : 0.0;
      }
    }
#pragma unroll
    for (int s = 0; s < UNROLL; ++s)
#pragma unroll
      for (int t = 0; t < TILES; ++t)
        if ((wg + WG * t) < mt_total)
#pragma unroll
          for (int u = 0; u < NT; ++u) dmma(acc[t][u], a[s][t], b[s][u]);
  }
  double* out = part + ((int64_t)blockIdx.x * RG + rg) * Mc * P;
#pragma unroll
  for (int t = 0; t < TILES; ++t) {
    const int mt = wg + WG * t;
    if (mt >= mt_total) continue;
    const int r = 8 * mt + (lane >> 2);
    if (r >= Mc) continue;
#pragma unroll
    for (int u = 0; u < NT; ++u)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = 8 * u + 2 * (lane & 3) + j;
        if (c < P) out[(int64_t)r * P + c] = acc[t][u][j];
      }
  }
}

// Row groups of one k_gram launch (as the kernel computes them).
inline int gram_groups(int Mc, int tiles_per_warp, int nwarp) {
  const int mt = (Mc + 7) / 8;
  const int wg = (mt + tiles_per_warp - 1) / tiles_per_warp;
  return 2 * wg > nwarp ? 1 : nwarp / wg;
}

// Sums the blocks' partials: a block of kRedWarps warps owns 32 consecutive entries of C; warp w
// adds the partials of blocks w, w + kRedWarps, ... (lane = entry, so each partial row is read as
// one 256-byte segment) and the warps' sums are combined in warp order, so the result is the same
// on every run.  32 warps: a narrow product leaves thousands of partials (148 blocks x 16 row
// groups) for few entries of C.
constexpr int kRedWarps = 32;
__global__ void __launch_bounds__(kRedWarps * 32) k_gram_reduce(const double* __restrict__ part,
                                                                int nblk, int M, int P, double alpha,
                                                                double beta, double* __restrict__ C,
                                                                int ldc, double* __restrict__ Acc,
                                                                int ldacc) {
  __shared__ double ws[kRedWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane;
  const int64_t mp = (int64_t)M * P;
  double s = 0.0;
  if (x < mp)
    for (int b = w; b < nblk; b += kRedWarps) s += part[b * mp + x];
  ws[w][lane] = s;
  __syncthreads();
  if (w == 0 && x < mp) {
    double t = ws[0][lane];
#pragma unroll
    for (int v = 1; v < kRedWarps; ++v) t += ws[v][lane];
    const int a = x / P, c = x - a * P;
    double* o = C + a + (int64_t)c * ldc;
    const double v = beta == 0.0 ? alpha * t : alpha * t + beta * *o;
    *o = v;
    if (Acc) Acc[a + (int64_t)c * ldacc] += v;
  }
}

// Shared row stride of the S slab: 8 NT + 4 doubles puts the four k-rows of one fragment load into
// distinct 32-byte bank groups.
constexpr int kRowsMaxM = 1280;     // rows of S held in shared memory per pass over A
constexpr int kRowsMaxM4 = 768;     // the same for 32-column slabs
constexpr int kRowsSelfMaxM = 960;  // the same beside the fused Gram product's reduction

template <int NT>
constexpr size_t rows_smem(int M) {
  return (size_t)M * (8 * NT + 4) * sizeof(double);
}

// What k_rows does beside its product.
struct RowsTail {
  const double* In;  // the beta term's block (ld ldi); Out itself unless given
  int ldi;
  double* Out2;      // second copy of the result (ld ldo2), or null
  int ldo2;
  double* part;      // partial Gram products Out^T Out, P x P per block, or null
};

// Out[i][c] = alpha sum_a A[i][a] S[a + c lds] + beta In[i][c] for Mc rows of S; warps stream 8-row
// tiles of A over the whole grid.  SELF: the tile's new rows also go, as they are in the accumulators
// (moved into operand layout by shuffles), into the warp's share of Out^T Out, so that the block
// orthonormalisation that follows a Gram-Schmidt pass needs no pass of its own (114 us at 120,011 rows
// and 512 columns on average, where the pass without it took 110 and the Gram product another 16).
template <int NT, bool SELF>
__global__ void __launch_bounds__(kThreads, 1) k_rows(const double* __restrict__ A, int lda,
                                                      const double* __restrict__ S, int lds,
                                                      int64_t n, int Mc, int P, double alpha,
                                                      double beta, double* Out, int ldo,
                                                      RowsTail tail) {
  extern __shared__ double ss[];  // [Mc][8 NT + 4]; SELF: then [warps][64 NT NT] for the reduction
  constexpr int SW = 8 * NT + 4;
  for (int x = threadIdx.x; x < Mc * 8 * NT; x += blockDim.x) {
    const int c = x / Mc, a = x - c * Mc;  // consecutive threads read one column of S
    ss[a * SW + c] = c < P ? S[a + (int64_t)c * lds] : 0.0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int kl = lane & 3;
  const int64_t tiles = (n + 7) / 8;
  const int64_t wstride = (int64_t)gridDim.x * (blockDim.x >> 5);
  double g[SELF ? NT : 1][SELF ? NT : 1][2];
  if constexpr (SELF) {
#pragma unroll
    for (int u = 0; u < NT; ++u)
#pragma unroll
      for (int v = 0; v < NT; ++v) g[u][v][0] = g[u][v][1] = 0.0;
  }
  for (int64_t tile = (int64_t)blockIdx.x * (blockDim.x >> 5) + wid; tile < tiles; tile += wstride) {
    const int64_t i = tile * 8 + (lane >> 2);
    const bool rin = i < n;
    const double* arow = A + (rin ? i : 0) * lda;
    double acc[NT][2];
#pragma unroll
    for (int u = 0; u < NT; ++u) acc[u][0] = acc[u][1] = 0.0;
    for (int k0 = 0; k0 < Mc; k0 += 4 * kUnroll) {
      double a[kUnroll];
#pragma unroll
      for (int s = 0; s < kUnroll; ++s) {
        const int k = k0 + 4 * s + kl;
        a[s] = (rin && k < Mc) ? __ldg(arow + k) : 0.0;
      }
#pragma unroll
      for (int s = 0; s < kUnroll; ++s) {
        const int k = k0 + 4 * s + kl;
        if (k0 + 4 * s < Mc) {
#pragma unroll
          for (int u = 0; u < NT; ++u)
            dmma(acc[u], a[s], k < Mc ? ss[k * SW + 8 * u + (lane >> 2)] : 0.0);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < NT; ++u)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = 8 * u + 2 * (lane & 3) + j;
        double o = 0.0;
        if (rin && c < P) {
          o = beta == 0.0 ? alpha * acc[u][j] : alpha * acc[u][j] + beta * tail.In[i * tail.ldi + c];
          Out[i * ldo + c] = o;
          if (tail.Out2) tail.Out2[i * tail.ldo2 + c] = o;
        }
        acc[u][j] = o;
      }
    if constexpr (SELF) {
      // operand element (row 4 h + (lane & 3), column 8 u + lane / 4) sits in lane
      // 4 row + (column % 8) / 2, place column % 2
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double w[NT];
        const int src = 4 * (4 * h + (lane & 3)) + (lane >> 3);
#pragma unroll
        for (int u = 0; u < NT; ++u) {
          const double x0 = __shfl_sync(0xffffffffu, acc[u][0], src);
          const double x1 = __shfl_sync(0xffffffffu, acc[u][1], src);
          w[u] = (lane >> 2) & 1 ? x1 : x0;
        }
#pragma unroll
        for (int u = 0; u < NT; ++u)
#pragma unroll
          for (int v = 0; v < NT; ++v) dmma(g[u][v], w[u], w[v]);
      }
    }
  }
  if constexpr (SELF) {
    // the warps' shares, added in warp order
    double* sg = ss + Mc * SW;
#pragma unroll
    for (int u = 0; u < NT; ++u)
#pragma unroll
      for (int v = 0; v < NT; ++v)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          sg[wid * 64 * NT * NT + (8 * u + (lane >> 2)) * 8 * NT + 8 * v + 2 * (lane & 3) + j] = g[u][v][j];
    __syncthreads();
    for (int x = threadIdx.x; x < 64 * NT * NT; x += blockDim.x) {
      const int r = x / (8 * NT), c = x - r * (8 * NT);
      if (r >= P || c >= P) continue;
      double t = 0.0;
      for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += sg[q * 64 * NT * NT + x];
      tail.part[(int64_t)blockIdx.x * P * P + r * P + c] = t;
    }
  }
}

// Shared memory of k_rows with the fused Gram product.
template <int NT>
constexpr size_t rows_self_smem(int M) {
  return rows_smem<NT>(M) + (size_t)(kThreads / 32) * 64 * NT * NT * sizeof(double);
}

// Orthonormalisation factor of a block W from its Gram matrix S = W^T W, given as nparts partial sums
// (nb x nb each, nb <= 16), in one block, so that a Lanczos step needs no host round trip.  With
// D = diag(S)^(-1/2) and D S D = R^T R (Cholesky), M = D R^(-1): W M is orthonormal to rounding times
// the conditioning of the scaled block, as for a factor from the eigenvectors of D S D.  A column
// whose pivot (the squared sine of its angle to the columns before it) is at most 1e-12, or whose
// diagonal is at most 1e-28 of the largest, is a lost direction: its column of M is zero and
// *rank_short is set.  One warp holds the matrix, lane = column; bound by the chain of nb square
// roots and divisions: measured 12 us with the sum of 148 partial products, where a Jacobi
// eigensolver took 88.
constexpr int kSvqbThreads = 1024;
__global__ void __launch_bounds__(kSvqbThreads) k_svqb_factor(const double* __restrict__ part,
                                                              int nparts, int nb,
                                                              double* __restrict__ M,
                                                              int* __restrict__ rank_short) {
  __shared__ double ps[4][256], A[16][17], R[16][17], rinv[16];
  const int tid = threadIdx.x;
  {  // four groups of threads add the partial sums q, q + 4, ...; then the groups in order
    const int x = tid & 255, q0 = tid >> 8;
    double t = 0.0;
    if (x < nb * nb)
#pragma unroll 8
      for (int q = q0; q < nparts; q += 4) t += part[(int64_t)q * nb * nb + x];
    ps[q0][x] = t;
  }
  __syncthreads();
  if (tid >= 32) return;
  for (int x = tid; x < nb * nb; x += 32)
    A[x / nb][x % nb] = ((ps[0][x] + ps[1][x]) + ps[2][x]) + ps[3][x];
  __syncwarp();
  const int c = tid;
  const bool in = c < nb;
  const double dc = in ? A[c][c] : 0.0;
  double dmax = dc;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(~0u, dmax, o));
  const bool live = in && dc > 1e-28 * dmax && dc > 1e-300;
  const double d = live ? 1.0 / sqrt(dc) : 0.0;
  // column c of the scaled matrix, from its upper triangle
  double a[16], r[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const double di = __shfl_sync(~0u, d, i);
    a[i] = (in && i <= c) ? A[i][c] * di * d : 0.0;
    r[i] = 0.0;
  }
  int lost = in && !live;
  // right-looking Cholesky: row i of R, then the trailing update of this lane's column
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    if (i < nb) {
      const double piv = __shfl_sync(~0u, a[i], i);
      const bool ok = piv > 1e-12;
      const double inv = ok ? rsqrt(piv) : 0.0;
      if (!ok && c == i) lost = 1;
      if (c == i) rinv[i] = inv;
      r[i] = (in && c >= i) ? a[i] * inv : 0.0;
      if (in) R[i][c] = r[i];
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j > i && j < nb && in && j <= c) a[j] = fma(-R[i][j], r[i], a[j]);
    }
  }
  // column c of R^(-1) by back substitution (zero for a lost direction)
  double x[16];
#pragma unroll
  for (int i = 15; i >= 0; --i) {
    x[i] = 0.0;
    if (i < nb && in && i <= c) {
      double t = i == c ? 1.0 : 0.0;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (j > i && j <= c) t = fma(-R[i][j], x[j], t);
      x[i] = t * rinv[i];
    }
  }
  const unsigned some = __ballot_sync(~0u, lost);
  if (some && tid == 0) *rank_short = 1;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const double di = __shfl_sync(~0u, d, i);
    if (i < nb && in) M[i + (int64_t)c * nb] = lost ? 0.0 : di * x[i];
  }
}

// One block per 32 vectors; the partial sums of G are added as in k_svqb_factor.
__global__ void __launch_bounds__(1024) k_krylov_residuals(const double* __restrict__ Y, int ldy, int nk,
                                                           const double* __restrict__ part, int nparts,
                                                           int P, double* __restrict__ rn2) {
  __shared__ double ps[4][256], G[256];
  const int tid = threadIdx.x;
  {
    const int x = tid & 255, q0 = tid >> 8;
    double t = 0.0;
    if (x < P * P)
#pragma unroll 8
      for (int q = q0; q < nparts; q += 4) t += part[(int64_t)q * P * P + x];
    ps[q0][x] = t;
  }
  __syncthreads();
  if (tid < P * P) G[tid] = ((ps[0][tid] + ps[1][tid]) + ps[2][tid]) + ps[3][tid];
  __syncthreads();
  const int j = blockIdx.x * 32 + (tid >> 5), a = tid & 31;
  if (j >= nk) return;
  double q = 0.0;
  if (a < P) {
    const double* y = Y + (int64_t)j * ldy;
    for (int e = 0; e < P; ++e) q = fma(G[a * P + e], y[e], q);
    q *= y[a];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(~0u, q, o);
  if (a == 0) rn2[j] = q;
}

__global__ void k_restart_matrix(double* __restrict__ T, int ld, const double* __restrict__ theta, int nk) {
  for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < ld * ld; x += gridDim.x * blockDim.x) {
    const int c = x / ld, r = x - c * ld;
    T[x] = r == c && r < nk ? theta[r] : 0.0;
  }
}

__global__ void k_add_cols(const double* __restrict__ src, int lds, int M, int P,
                           double* __restrict__ dst, int ldd) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= M * P) return;
  const int c = x / M, a = x - c * M;
  dst[a + (int64_t)c * ldd] += src[a + (int64_t)c * lds];
}

// The dynamic shared-memory limits are set once per process to the largest size any launch uses,
// so concurrent contexts never race on them.
std::once_flag g_attr_once;
void set_attributes() {
  std::call_once(g_attr_once, [] {
    cudaFuncSetAttribute(k_rows<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rows_smem<1>(kRowsMaxM));
    cudaFuncSetAttribute(k_rows<2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rows_smem<2>(kRowsMaxM));
    cudaFuncSetAttribute(k_rows<4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rows_smem<4>(kRowsMaxM4));
    cudaFuncSetAttribute(k_rows<1, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rows_self_smem<1>(kRowsSelfMaxM));
    cudaFuncSetAttribute(k_rows<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)rows_self_smem<2>(kRowsSelfMaxM));
  });
}

}  // namespace

void svqb_factor(const double* part, int nparts, int nb, double* M, int* rank_short,
                 cudaStream_t s) {
  note_launch();
  k_svqb_factor<<<1, kSvqbThreads, 0, s>>>(part, nparts, nb, M, rank_short);
}

int64_t proj_gram_scratch(int M, int P) {
  // blocks x row groups x Mc <= kBlocks x kGramSlab for every slab width (groups x tiles <= 96)
  (void)M;
  return (int64_t)kBlocks * kGramSlab * P;
}

bool proj_gram(const double* A, int lda, const double* B, int ldb, int64_t n, int M, int P,
               double alpha, double beta, double* C, int ldc, double* part, cudaStream_t s,
               double* Acc, int ldacc) {
  if (M <= 0 || P <= 0) return true;
  if (P > 16 || lda < M || ldb < P) return false;
  int nblk = kBlocks;
  if (n < (int64_t)nblk * 64) nblk = (int)std::max<int64_t>(1, (n + 63) / 64);
  for (int a0 = 0; a0 < M; a0 += kGramSlab) {
    const int Mc = std::min(kGramSlab, M - a0);
    // up to 16 tiles of C: 16 warps, one tile each, eight k-steps in flight; up to 64 tiles: 32
    // warps, two tiles each, four k-steps; wider: 16 warps, six tiles each, two k-steps (measured
    // on 380k rows, P = 16: 0.39 ms against 0.47 ms at M = 512 for the middle form, and 0.50
    // against 0.55 ms at M = 672 for the wide one)
    const int form = Mc <= 8 * kGramWarps ? 0 : (Mc <= 8 * 2 * 32 ? 1 : 2);
    const int nparts = nblk * (form == 0   ? gram_groups(Mc, 1, kGramWarps)
                               : form == 1 ? gram_groups(Mc, 2, 32)
                                           : gram_groups(Mc, kGramTiles, kGramWarps));
    note_launch();
    if (form == 0) {
      if (P <= 8) k_gram<1, 1, 8, kGramWarps><<<nblk, kGramThreads, 0, s>>>(A + a0, lda, B, ldb, n, Mc, P, part);
      else k_gram<2, 1, 8, kGramWarps><<<nblk, kGramThreads, 0, s>>>(A + a0, lda, B, ldb, n, Mc, P, part);
    } else if (form == 1) {
      if (P <= 8) k_gram<1, 2, 4, 32><<<nblk, 1024, 0, s>>>(A + a0, lda, B, ldb, n, Mc, P, part);
      else k_gram<2, 2, 4, 32><<<nblk, 1024, 0, s>>>(A + a0, lda, B, ldb, n, Mc, P, part);
    } else {
      if (P <= 8)
        k_gram<1, kGramTiles, kGramUnroll, kGramWarps><<<nblk, kGramThreads, 0, s>>>(A + a0, lda, B, ldb, n, Mc, P, part);
      else
        k_gram<2, kGramTiles, kGramUnroll, kGramWarps><<<nblk, kGramThreads, 0, s>>>(A + a0, lda, B, ldb, n, Mc, P, part);
    }
    note_launch();
    k_gram_reduce<<<(Mc * P + 31) / 32, kRedWarps * 32, 0, s>>>(part, nparts, Mc, P, alpha, beta,
                                                                 C + a0, ldc, Acc ? Acc + a0 : nullptr,
                                                                 ldacc);
  }
  return true;
}

void proj_rows(const double* A, int lda, const double* S, int lds, int64_t n, int M, int P,
               double alpha, double beta, double* Out, int ldo, cudaStream_t s, const double* In,
               int ldi, double* Out2, int ldo2) {
  if (n <= 0 || P <= 0) return;
  set_attributes();
  const int64_t tiles = (n + 7) / 8;
  const int g = (int)std::min<int64_t>(kBlocks, (tiles + 31) / 32);
  // 32-column slabs when S's rows fit beside them in shared memory: half the passes over A
  const int cw = (P > 16 && M <= kRowsMaxM4) ? 32 : 16;
  for (int c0 = 0; c0 < P; c0 += cw) {
    const int pc = std::min(cw, P - c0);
    double* Oc = Out + c0;
    // slabs of S rows; every slab after the first adds into Out
    for (int a0 = 0; a0 < std::max(M, 1); a0 += kRowsMaxM) {
      const int Mc = std::min(kRowsMaxM, M - a0);
      const double* Sc = S + (int64_t)c0 * lds + a0;
      const double bt = a0 == 0 ? beta : 1.0;
      const bool last = a0 + kRowsMaxM >= M;
      const RowsTail t{a0 == 0 && In ? In + c0 : Oc, a0 == 0 && In ? ldi : ldo,
                       last && Out2 ? Out2 + c0 : nullptr, ldo2, nullptr};
      note_launch();
      if (pc > 16)
        k_rows<4, false><<<g, kThreads, rows_smem<4>(std::max(Mc, 1)), s>>>(A + a0, lda, Sc, lds, n, Mc,
                                                                            pc, alpha, bt, Oc, ldo, t);
      else if (pc <= 8)
        k_rows<1, false><<<g, kThreads, rows_smem<1>(std::max(Mc, 1)), s>>>(A + a0, lda, Sc, lds, n, Mc,
                                                                            pc, alpha, bt, Oc, ldo, t);
      else
        k_rows<2, false><<<g, kThreads, rows_smem<2>(std::max(Mc, 1)), s>>>(A + a0, lda, Sc, lds, n, Mc,
                                                                            pc, alpha, bt, Oc, ldo, t);
    }
  }
}

int proj_rows_self(const double* A, int lda, const double* S, int lds, int64_t n, int M, int P,
                   double* W, int ldw, double* part, cudaStream_t s) {
  if (n <= 0 || P <= 0 || P > 16 || M <= 0 || M > kRowsSelfMaxM) return 0;
  set_attributes();
  const int g = (int)std::min<int64_t>(kBlocks, ((n + 7) / 8 + 31) / 32);
  const RowsTail t{W, ldw, nullptr, 0, part};
  note_launch();
  if (P <= 8)
    k_rows<1, true><<<g, kThreads, rows_self_smem<1>(M), s>>>(A, lda, S, lds, n, M, P, -1.0, 1.0, W, ldw, t);
  else
    k_rows<2, true><<<g, kThreads, rows_self_smem<2>(M), s>>>(A, lda, S, lds, n, M, P, -1.0, 1.0, W, ldw, t);
  return g;
}

void krylov_residuals(const double* Y, int ldy, int nk, const double* part, int nparts, int P,
                      double* rn2, cudaStream_t s) {
  if (nk <= 0) return;
  note_launch();
  k_krylov_residuals<<<(nk + 31) / 32, 1024, 0, s>>>(Y, ldy, nk, part, nparts, P, rn2);
}

void restart_matrix(double* T, int ld, const double* theta, int nk, cudaStream_t s) {
  note_launch();
  k_restart_matrix<<<std::min(592, (ld * ld + 255) / 256), 256, 0, s>>>(T, ld, theta, nk);
}

void add_cols(const double* src, int lds, int M, int P, double* dst, int ldd, cudaStream_t s) {
  if (M <= 0 || P <= 0) return;
  note_launch();
  k_add_cols<<<(M * P + 255) / 256, 256, 0, s>>>(src, lds, M, P, dst, ldd);
}

void gram_sum(const double* part, int nparts, int M, int P, double* C, int ldc, cudaStream_t s) {
  note_launch();
  k_gram_reduce<<<(M * P + 31) / 32, kRedWarps * 32, 0, s>>>(part, nparts, M, P, 1.0, 0.0, C, ldc,
                                                              nullptr, 0);
}

}  // namespace vhci
