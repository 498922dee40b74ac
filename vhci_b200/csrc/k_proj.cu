// FP64 tensor-core projections for the block Lanczos eigensolver (the Gram-Schmidt passes, the
// block orthonormalisation and the Rayleigh-Ritz rotations).  The reference eigensolver (Spectra's
// implicitly restarted Lanczos, Ham.cpp:347-370) does these with Eigen's dense products; here they
// are skinny products over the whole basis, written for B200's FP64 tensor pipe (DMMA,
// mma.sync.m8n8k4.f64).  Both read the tall operand once, straight from global memory into the
// DMMA fragment registers, 32 bytes a lane: what a lane holds of four (or two) adjacent columns is
// its element of four fragments, so that a fragment's columns lie four apart in the operand.  An
// 8-byte load a lane visits one cache line for every 32 bytes, and the line lookups of the first
// cache level were the limit (84 % of its peak at 42 % of the memory's bandwidth, 100,000 rows).
//
//   proj_gram:  C = alpha * A^T B + beta * C   A: n x M, B: n x P (row-major), C: M x P col-major,
//               P <= 16.  A persistent grid splits the n rows over the blocks; each warp keeps
//               the partial products of its 16 or 32 rows of C in registers; the blocks' partials
//               go to scratch and a second kernel sums them in block order, so the result does not
//               depend on scheduling.
//   proj_rows:  Out = alpha * A S + beta * In    A: n x M row-major, S: M x P col-major,
//               Out: n x P row-major.  Each block holds a 16- or 32-column slab of S in shared memory
//               and its warps stream 8-row tiles of A.  proj_rows_self also forms Out^T Out.
//
// A Lanczos step reads the basis twice (coefficients, update).  Three passes with the first two fused
// over 128-row chunks took 240 + 110 us of projections at 120,011 rows and 512 columns on average,
// 44 us at 24,000 rows and 150 columns; with 8-byte loads 150 + 110 and 16 + 13 us, now 99 + 100 and 13 +
// 11 us (the bytes of one pass take 75 us at 120,011 rows, and its products 52 us at 37 TFLOP/s).
//
// Fragment layouts of m8n8k4 (row.col): A[m][k] sits in lane 4 m + k, B[k][n] in lane 4 n + k,
// D[m][n] in lane 4 m + n / 2 (element n % 2).
#include <algorithm>
#include <cstdint>
#include <mutex>

#include "chain.cuh"
#include "ops.h"

namespace vhci {

namespace {

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

constexpr int kThreads = 512;       // proj_rows: 16 warps with up to 128 registers each, one block per SM
constexpr int kAhead = 4;           // proj_rows: loads of 16 columns in flight per warp
constexpr int kBlocks = 148;
constexpr int kGramSlab = 764;      // columns of A in one launch of k_gram: 24 tiles of 32 with any skew

// Four adjacent doubles at p, of which those with first <= k < last (k: the index of p[0]) are wanted.
// wide: p is 32-byte aligned, and the four are one load; a sector that holds a wanted element lies
// within its allocation, and mask4 clears the others before they are used.
__device__ __forceinline__ void load4(double (&v)[4], const double* p, int k, int first, int last,
                                      bool wide) {
  v[0] = v[1] = v[2] = v[3] = 0.0;
  if (wide) {
    if (k + 3 >= first && k < last)
      asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                   : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                   : "l"(p));
  } else {
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (k + s >= first && k + s < last) v[s] = p[s];
  }
}

__device__ __forceinline__ void mask4(double (&v)[4], int k, int first, int last) {
  if (k < first || k + 3 >= last) {
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (k + s < first || k + s >= last) v[s] = 0.0;
  }
}

// How far a pointer lies past a 32-byte boundary, in doubles, where its rows all start alike; 0 and
// wide = false where they do not.
inline int row_skew(const double* A, int lda, bool* wide) {
  *wide = lda % 4 == 0;
  return *wide ? (int)(reinterpret_cast<uintptr_t>(A) / sizeof(double) % 4) : 0;
}

// Partial A^T B over this block's rows for Mc columns of A (A points skew columns before the first).
// The columns are dealt in tiles of 8 CT to a group of WG warps, one tile a warp; the block's warps
// form NWARP / WG groups, which take turns over the block's rows in steps of 4 UNROLL rows, so a
// narrow C (few tiles) still keeps every warp streaming.  A lane loads CT adjacent columns of its row:
// its elements of CT fragments, fragment t holding the columns t, t + CT, ... of the tile; B's columns
// are taken NT apart likewise.  Each step's registers are loaded anew, for the next round, as soon as
// its products are issued, so that loads and products of one warp overlap.
// Block x writes its partial to part[x] (Mc x P, a-major).
template <int NT, int CT, int UNROLL, int NWARP>
__global__ void __launch_bounds__(NWARP * 32, 1) k_gram(const double* A, int lda,
                                                    const double* B, int ldb,
                                                    int64_t n, int Mc, int P, int skew, bool wide,
                                                    bool bwide, double* __restrict__ part) {
  chain_wait();
  static_assert(CT == 2 || CT == 4, "");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int last = skew + Mc;
  const int WG = (last + 8 * CT - 1) / (8 * CT);
  const int RG = NWARP / WG;
  const int rg = wid / WG, wg = wid - rg * WG;  // warps with rg >= RG have no rows
  const int64_t per = ((n + gridDim.x - 1) / gridDim.x + 3) & ~int64_t(3);
  const int64_t r0 = (int64_t)blockIdx.x * per, r1 = min(n, r0 + per);
  double acc[CT][NT][2];
#pragma unroll
  for (int t = 0; t < CT; ++t)
#pragma unroll
    for (int u = 0; u < NT; ++u) acc[t][u][0] = acc[t][u][1] = 0.0;
  const int acol = 8 * CT * wg + CT * (lane >> 2);  // from A, so the lane's columns start at acol - skew
  const bool ain = acol + CT - 1 >= skew && acol < last, aall = acol >= skew && acol + CT <= last;
  const int bcol = NT * (lane >> 2);
  const int kl = lane & 3;
  double a[UNROLL][CT], b[UNROLL][NT];
  auto load = [&](int s, int64_t i) {
    const bool rin = i < r1;
    const double* p = A + i * lda + acol;
#pragma unroll
    for (int t = 0; t < CT; ++t) a[s][t] = 0.0;
    if (wide) {
      if (rin && ain) {
        if constexpr (CT == 4) {
          asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];"
                       : "=d"(a[s][0]), "=d"(a[s][1]), "=d"(a[s][2]), "=d"(a[s][3])
                       : "l"(p));
        } else {
          asm volatile("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(a[s][0]), "=d"(a[s][1]) : "l"(p));
        }
      }
    } else {
#pragma unroll
      for (int t = 0; t < CT; ++t)
        if (rin && acol + t < last) a[s][t] = p[t];
    }
    const double* q = B + i * ldb + bcol;
#pragma unroll
    for (int u = 0; u < NT; ++u) b[s][u] = 0.0;
    if (NT == 2 && bwide) {
      if (rin) asm volatile("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(b[s][0]), "=d"(b[s][NT - 1]) : "l"(q));
    } else {
#pragma unroll
      for (int u = 0; u < NT; ++u)
        if (rin && bcol + u < P) b[s][u] = q[u];
    }
  };
  const int64_t first = rg < RG ? r0 + 4 * UNROLL * rg + kl : r1 + kl;
#pragma unroll
  for (int s = 0; s < UNROLL; ++s) load(s, first + 4 * s);
  for (int64_t k0 = first; k0 - kl < r1; k0 += 4 * UNROLL * RG) {
#pragma unroll
    for (int s = 0; s < UNROLL; ++s) {
      if (wide && !aall)
#pragma unroll
        for (int t = 0; t < CT; ++t)
          if (acol + t < skew || acol + t >= last) a[s][t] = 0.0;
#pragma unroll
      for (int t = 0; t < CT; ++t)
#pragma unroll
        for (int u = 0; u < NT; ++u) dmma(acc[t][u], a[s][t], b[s][u]);
      load(s, k0 + 4 * UNROLL * RG + 4 * s);
    }
  }
  if (RG > 1) {  // the groups' sums, added in order by the first
    constexpr int kTile = CT * NT * 2;
    extern __shared__ double sg[];  // [RG - 1][WG][kTile][32]
    double* own = sg + ((rg - 1) * WG + wg) * kTile * 32 + lane;
    if (rg > 0 && rg < RG)
#pragma unroll
      for (int x = 0; x < kTile; ++x) own[x * 32] = acc[x / (2 * NT)][x / 2 % NT][x % 2];
    __syncthreads();
    if (rg == 0)
      for (int q = 0; q < RG - 1; ++q)
#pragma unroll
        for (int x = 0; x < kTile; ++x)
          acc[x / (2 * NT)][x / 2 % NT][x % 2] += sg[((q * WG + wg) * kTile + x) * 32 + lane];
  }
  if (rg > 0) return;
  double* out = part + (int64_t)blockIdx.x * Mc * P;
#pragma unroll
  for (int t = 0; t < CT; ++t) {
    const int r = acol + t - skew;
    if (r < 0 || r >= Mc) continue;
#pragma unroll
    for (int u = 0; u < NT; ++u)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int c = NT * (2 * (lane & 3) + j) + u;
        if (c < P) out[(int64_t)r * P + c] = acc[t][u][j];
      }
  }
}

template <int CT, int UNROLL, int NWARP>
void launch_gram(const double* A, int lda, const double* B, int ldb, int64_t n, int nblk, int Mc, int P,
                 int skew, bool wide, double* part, cudaStream_t s) {
  // all of a row's 16 columns of B as pairs
  const bool bwide = P == 16 && ldb % 2 == 0 && reinterpret_cast<uintptr_t>(B) % 16 == 0;
  const int wg = (skew + Mc + 8 * CT - 1) / (8 * CT);
  const size_t tiles = (size_t)(NWARP / wg - 1) * wg;  // of the groups beside the first: 12 of 32 columns, 15 of 16
  const size_t smem = tiles * 8 * CT * (P <= 8 ? 8 : 16) * sizeof(double);
  note_launch();
  if (P <= 8)
    launch_chained(k_gram<1, CT, UNROLL, NWARP>, nblk, NWARP * 32, smem, s, A - skew, lda, B, ldb, n, Mc, P, skew, wide,
                                                                bwide, part);
  else
    launch_chained(k_gram<2, CT, UNROLL, NWARP>, nblk, NWARP * 32, smem, s, A - skew, lda, B, ldb, n, Mc, P, skew, wide,
                                                                bwide, part);
}

// Sums the blocks' partials: a block of kRedWarps warps owns 32 consecutive entries of C; warp w
// adds the partials of blocks w, w + kRedWarps, ... (lane = entry, so each partial row is read as
// one 256-byte segment) and the warps' sums are combined in warp order, so the result is the same
// on every run.
constexpr int kRedWarps = 32;
__global__ void __launch_bounds__(kRedWarps * 32) k_gram_reduce(const double* part,
                                                                int nblk, int M, int P, double alpha,
                                                                double beta, double* __restrict__ C,
                                                                int ldc, double* __restrict__ Acc,
                                                                int ldacc) {
  chain_wait();
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

constexpr int kRowsMaxM = 1280;     // rows of S held in shared memory per pass over A
constexpr int kRowsMaxM4 = 768;     // the same for 32-column slabs
constexpr int kRowsSelfMaxM = 960;  // the same beside the fused Gram product's reduction

// Place of element (k, c) of the S slab in shared memory.  A fragment load takes row 16 j + 4 q + s of
// column pairs c, c + 1 (NT = 2; single columns for 1, two pairs for 4), q and c / NT differing over the
// lanes: the rows are rotated in 32-byte groups, or padded, such that these lie in distinct banks.
template <int NT>
__host__ __device__ constexpr int s_place(int k, int c) {
  return NT == 1   ? k * 9 + c
         : NT == 2 ? k * 16 + (c ^ ((k & 12) | ((k & 1) << 1)))
                   : k * 32 + (c ^ (((k & 4) << 1) | ((k & 8) >> 2)));
}

template <int NT>
constexpr size_t rows_smem(int M) {
  return (size_t)((M + 3 + 15) / 16 * 16) * (NT == 1 ? 9 : 8 * NT) * sizeof(double);
}

// What k_rows does beside its product.
struct RowsTail {
  const double* In;  // the beta term's block (ld ldi); Out itself unless given
  int ldi;
  double* Out2;      // second copy of the result (ld ldo2), or null
  int ldo2;
  double* part;      // partial Gram products Out^T Out, P x P per block, or null
};

// Out[i][c] = alpha sum_a A[i][a] S[a + c lds] + beta In[i][c] for Mc rows of S (A points skew columns
// before the first; vec: rows of Out, In and Out2 are 16-byte aligned and P = 8 NT); warps stream 8-row
// tiles of A over the whole grid, 16 columns in one 32-byte load a lane, each load issued as soon as its
// registers' products are (the next tile's first ones too).  Fragment u of
// the result holds the columns u, u + NT, ..., so that a lane's elements of a row are adjacent.
// SELF: the tile's new rows also go, as they are in the accumulators (moved into operand layout by
// shuffles), into the warp's share of Out^T Out, so that the block orthonormalisation that follows a
// Gram-Schmidt pass needs no pass of its own.  Updates of 120,011 rows by 320 to 672
// columns take 100 us (110 with 8-byte loads of 32 warps and the tiles of the last round on a third of the
// SMs); a 32-column rotation of 672 columns takes 197 us, of which the tensor pipe needs 140 (231 before).
template <int NT, bool SELF>
__global__ void __launch_bounds__(kThreads, 1) k_rows(const double* A, int lda,
                                                      const double* S, int lds,
                                                      int64_t n, int Mc, int P, int skew, bool wide,
                                                      bool vec, double alpha, double beta, double* Out,
                                                      int ldo, RowsTail tail) {
  chain_wait();
  extern __shared__ __align__(16) double ss[];  // the S slab; SELF: then [warps][64 NT NT] for the reduction
  const int last = skew + Mc, Mr = (last + 15) / 16 * 16;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int kl = lane & 3;
  const int64_t tiles = (n + 7) / 8;
  const int64_t wstride = (int64_t)gridDim.x * (blockDim.x >> 5);
  // a round's tiles go over the blocks first, so that the last round is spread over all of them
  const int64_t tile0 = (int64_t)wid * gridDim.x + blockIdx.x;
  double a[kAhead][4];
  {
    const int64_t i = tile0 * 8 + (lane >> 2);
#pragma unroll
    for (int h = 0; h < kAhead; ++h)
      load4(a[h], A + (i < n ? i : 0) * lda + 16 * h + 4 * kl, 16 * h + 4 * kl, skew, i < n ? last : 0, wide);
  }
  for (int c = wid; c < 8 * NT; c += blockDim.x >> 5) {
    const double* Sc = S - skew + (int64_t)c * lds;
#pragma unroll 4
    for (int k = lane; k < Mr; k += 32)
      ss[s_place<NT>(k, c)] = c < P && k >= skew && k < last ? Sc[k] : 0.0;
  }
  __syncthreads();
  const int c0 = 2 * NT * kl;  // the lane's columns of the result: c0 + NT j + u
  double g[SELF ? NT : 1][SELF ? NT : 1][2];
  if constexpr (SELF) {
#pragma unroll
    for (int u = 0; u < NT; ++u)
#pragma unroll
      for (int v = 0; v < NT; ++v) g[u][v][0] = g[u][v][1] = 0.0;
  }
  for (int64_t tile = tile0; tile < tiles; tile += wstride) {
    const int64_t i = tile * 8 + (lane >> 2);
    const bool rin = i < n;
    const int64_t inext = i + 8 * wstride;
    const double* arow = A + (rin ? i : 0) * lda + 4 * kl;
    const double* anext = A + (inext < n ? inext : 0) * lda + 4 * kl;
    const int rlast = rin ? last : 0, nlast = inext < n ? last : 0;
    double acc[NT][2];
#pragma unroll
    for (int u = 0; u < NT; ++u) acc[u][0] = acc[u][1] = 0.0;
    for (int k0 = 0; k0 < Mr; k0 += 16 * kAhead) {
      const bool more = k0 + 16 * kAhead < Mr;
#pragma unroll
      for (int h = 0; h < kAhead; ++h) {
        mask4(a[h], k0 + 16 * h + 4 * kl, skew, rlast);
        const int k = k0 + 16 * h + 4 * kl;
        if (k0 + 16 * h < Mr)
#pragma unroll
          for (int s = 0; s < 4; ++s) {
            if constexpr (NT == 1) {
              dmma(acc[0], a[h][s], ss[s_place<1>(k + s, lane >> 2)]);
            } else {
#pragma unroll
              for (int u = 0; u < NT; u += 2) {
                const double2 v =
                    *reinterpret_cast<const double2*>(ss + s_place<NT>(k + s, NT * (lane >> 2) + u));
                dmma(acc[u], a[h][s], v.x);
                dmma(acc[u + 1], a[h][s], v.y);
              }
            }
          }
        const int kn = (more ? k0 + 16 * kAhead : 0) + 16 * h;
        load4(a[h], (more ? arow : anext) + kn, kn + 4 * kl, skew, more ? rlast : nlast, wide);
      }
    }
    if (vec) {
#pragma unroll
      for (int x = 0; x < 2 * NT; x += 2) {  // place x of the lane's row segment: j = x / NT, u = x % NT
        double2 o = make_double2(0.0, 0.0);
        if (rin) {
          o.x = alpha * acc[x % NT][x / NT];
          o.y = alpha * acc[(x + 1) % NT][(x + 1) / NT];
          if (beta != 0.0) {
            const double2 v = *reinterpret_cast<const double2*>(tail.In + i * tail.ldi + c0 + x);
            o.x += beta * v.x;
            o.y += beta * v.y;
          }
          *reinterpret_cast<double2*>(Out + i * ldo + c0 + x) = o;
          if (tail.Out2) *reinterpret_cast<double2*>(tail.Out2 + i * tail.ldo2 + c0 + x) = o;
        }
        acc[x % NT][x / NT] = o.x;
        acc[(x + 1) % NT][(x + 1) / NT] = o.y;
      }
    } else {
#pragma unroll
      for (int u = 0; u < NT; ++u)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int c = c0 + NT * j + u;
          double o = 0.0;
          if (rin && c < P) {
            o = beta == 0.0 ? alpha * acc[u][j] : alpha * acc[u][j] + beta * tail.In[i * tail.ldi + c];
            Out[i * ldo + c] = o;
            if (tail.Out2) tail.Out2[i * tail.ldo2 + c] = o;
          }
          acc[u][j] = o;
        }
    }
    if constexpr (SELF) {
      // operand element (row 4 h + (lane & 3), place lane / 4 of fragment u) sits in lane
      // 4 row + place / 2, element place % 2
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
    double* sg = ss + Mr * (NT == 1 ? 9 : 8 * NT);
#pragma unroll
    for (int u = 0; u < NT; ++u)
#pragma unroll
      for (int v = 0; v < NT; ++v)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          sg[wid * 64 * NT * NT + (NT * (lane >> 2) + u) * 8 * NT + NT * (2 * (lane & 3) + j) + v] =
              g[u][v][j];
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

inline bool pair_rows(const double* p, int ld) {
  return ld % 2 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0;
}

template <int NT, bool SELF>
void launch_rows(const double* A, int lda, const double* S, int lds, int64_t n, int Mc, int P, double alpha,
                 double beta, double* Out, int ldo, const RowsTail& t, int blocks, cudaStream_t s) {
  bool wide;
  const int skew = row_skew(A, lda, &wide);
  const bool vec = P == 8 * NT && pair_rows(Out, ldo) && (beta == 0.0 || pair_rows(t.In, t.ldi)) &&
                   (!t.Out2 || pair_rows(t.Out2, t.ldo2));
  const size_t smem = SELF ? rows_self_smem<NT>(Mc) : rows_smem<NT>(Mc);
  note_launch();
  launch_chained(k_rows<NT, SELF>, blocks, kThreads, smem, s, A - skew, lda, S, lds, n, Mc, P, skew, wide, vec, alpha,
                                                  beta, Out, ldo, t);
}

// Orthonormalisation factor of a block W from its Gram matrix S = W^T W, given as nparts partial sums
// (nb x nb each, nb <= 16), in one block, so that a Lanczos step needs no host round trip.  With
// D = diag(S)^(-1/2) and D S D = R^T R (Cholesky), M = D R^(-1): W M is orthonormal to rounding times
// the conditioning of the scaled block, as for a factor from the eigenvectors of D S D.  A column
// whose pivot (the squared sine of its angle to the columns before it) is at most 1e-12, or whose
// diagonal is at most 1e-28 of the largest, is a lost direction: its column of M is zero and
// *rank_short is set.  One warp holds the matrix, lane = column; bound by the chain of nb square
// roots and divisions: measured 11 us with the sum of 148 partial products, where a Jacobi
// eigensolver took 88.
constexpr int kSvqbThreads = 1024;
__global__ void __launch_bounds__(kSvqbThreads) k_svqb_factor(const double* part,
                                                              int nparts, int nb,
                                                              double* __restrict__ M,
                                                              int* __restrict__ rank_short) {
  chain_wait();
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
__global__ void __launch_bounds__(1024) k_krylov_residuals(const double* Y, int ldy, int nk,
                                                           const double* part, int nparts,
                                                           int P, double* __restrict__ rn2) {
  chain_wait();
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

__global__ void k_restart_matrix(double* __restrict__ T, int ld, const double* theta, int nk) {
  chain_wait();
  for (int x = blockIdx.x * blockDim.x + threadIdx.x; x < ld * ld; x += gridDim.x * blockDim.x) {
    const int c = x / ld, r = x - c * ld;
    T[x] = r == c && r < nk ? theta[r] : 0.0;
  }
}

__global__ void k_add_cols(const double* src, int lds, int M, int P,
                           double* __restrict__ dst, int ldd) {
  chain_wait();
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
  launch_chained(k_svqb_factor, 1, kSvqbThreads, 0, s, part, nparts, nb, M, rank_short);
}

int64_t proj_gram_scratch(int M, int P) {
  // a partial of at most kGramSlab x P a block
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
    bool wide;
    const int skew = row_skew(A + a0, lda, &wide);
    // Up to 128 columns: tiles of 16, so that the warps of a narrow C share the rows among at least two
    // groups.  Wider: tiles of 32, one a warp; 24 warps where 16 would leave 4 or more of them idle
    // (9 to 12 tiles), or are too few.  At 120,011 rows and P = 16: 88 us for 13 to 16 tiles on average,
    // 107 for 17 to 21 (130 and 134 with each round's loads waited for before its products).
    const int t32 = (skew + Mc + 31) / 32;
    if (skew + Mc <= 128) launch_gram<2, 8, 16>(A + a0, lda, B, ldb, n, nblk, Mc, P, skew, wide, part, s);
    else if (t32 <= 8 || (t32 > 12 && t32 <= 16))
      launch_gram<4, 4, 16>(A + a0, lda, B, ldb, n, nblk, Mc, P, skew, wide, part, s);
    else
      launch_gram<4, 2, 24>(A + a0, lda, B, ldb, n, nblk, Mc, P, skew, wide, part, s);
    note_launch();
    launch_chained(k_gram_reduce, (Mc * P + 31) / 32, kRedWarps * 32, 0, s, part, nblk, Mc, P, alpha, beta,
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
  const int g = (int)std::min<int64_t>(kBlocks, (tiles + 15) / 16);
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
      if (pc > 16) launch_rows<4, false>(A + a0, lda, Sc, lds, n, Mc, pc, alpha, bt, Oc, ldo, t, g, s);
      else if (pc <= 8) launch_rows<1, false>(A + a0, lda, Sc, lds, n, Mc, pc, alpha, bt, Oc, ldo, t, g, s);
      else launch_rows<2, false>(A + a0, lda, Sc, lds, n, Mc, pc, alpha, bt, Oc, ldo, t, g, s);
    }
  }
}

int proj_rows_self(const double* A, int lda, const double* S, int lds, int64_t n, int M, int P,
                   double* W, int ldw, double* part, cudaStream_t s) {
  if (n <= 0 || P <= 0 || P > 16 || M <= 0 || M > kRowsSelfMaxM) return 0;
  set_attributes();
  const int g = (int)std::min<int64_t>(kBlocks, ((n + 7) / 8 + 15) / 16);
  const RowsTail t{W, ldw, nullptr, 0, part};
  if (P <= 8) launch_rows<1, true>(A, lda, S, lds, n, M, P, -1.0, 1.0, W, ldw, t, g, s);
  else launch_rows<2, true>(A, lda, S, lds, n, M, P, -1.0, 1.0, W, ldw, t, g, s);
  return g;
}

void krylov_residuals(const double* Y, int ldy, int nk, const double* part, int nparts, int P,
                      double* rn2, cudaStream_t s) {
  if (nk <= 0) return;
  note_launch();
  launch_chained(k_krylov_residuals, (nk + 31) / 32, 1024, 0, s, Y, ldy, nk, part, nparts, P, rn2);
}

void restart_matrix(double* T, int ld, const double* theta, int nk, cudaStream_t s) {
  note_launch();
  launch_chained(k_restart_matrix, std::min(592, (ld * ld + 255) / 256), 256, 0, s, T, ld, theta, nk);
}

void add_cols(const double* src, int lds, int M, int P, double* dst, int ldd, cudaStream_t s) {
  if (M <= 0 || P <= 0) return;
  note_launch();
  launch_chained(k_add_cols, (M * P + 255) / 256, 256, 0, s, src, lds, M, P, dst, ldd);
}

void gram_sum(const double* part, int nparts, int M, int P, double* C, int ldc, cudaStream_t s) {
  note_launch();
  launch_chained(k_gram_reduce, (M * P + 31) / 32, kRedWarps * 32, 0, s, part, nparts, M, P, 1.0, 0.0, C, ldc,
                                                              nullptr, 0);
}

}  // namespace vhci
