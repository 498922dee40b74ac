// Hamiltonian kernels: the connection-driven sparse build (replacing the reference's O(N^2) pair
// loop, Ham.cpp:228-326), the SpMM that drives the eigensolver, and the Davidson vector helpers.
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <string>

#include "chain.cuh"
#include "conn.cuh"
#include "ops.h"
#include "rowprod.cuh"

namespace vhci {

namespace {

inline int grid_for(int64_t n, int threads, int max_blocks = 148 * 16) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (int)b;
}

}  // namespace

namespace {

// One warp per row: the states that the row's state is connected to (conn.cuh), in the walk's fixed
// order, counted (and kept in `stage` when it has room) or written with their matrix elements
// (FILL).  Row i is basis state row0 + stride i; columns are basis indices.  Blocks of four rows, no
// loop: rows differ in work by their excited modes, and the hardware evens that out.
template <int W, bool FILL>
__global__ void __launch_bounds__(kWalkThreads) k_hbuild(
    const uint64_t* __restrict__ keys, int64_t row0, int64_t stride, int64_t n, KeyLayout L,
    HashView basis, ConnDev cd, int32_t* __restrict__ rowcnt, StageView stage,
    const int64_t* __restrict__ rowptr, int32_t* __restrict__ col, double* __restrict__ val,
    float* __restrict__ valf) {
  __shared__ uint32_t s_binom[kBinomElems];
  __shared__ WalkScratch<false> s_walk[kWalkWarps];
  fill_binom(s_binom);
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)kWalkWarps + (threadIdx.x >> 5);
  if (i >= n) return;
  uint64_t k[W];
  load_key<W>(keys, row0 + stride * i, k);
  const int64_t pos = FILL ? rowptr[i] : 0;
  int cnt = 0;
  walk_connections<W>(cd, basis, k, L, s_walk[threadIdx.x >> 5], s_binom, nullptr, [&](int64_t j, uint32_t u) {
    const unsigned b = __ballot_sync(0xffffffffu, j >= 0);
    if (FILL) {
      if (j >= 0) {
        const int64_t p = pos + cnt + __popc(b & lanemask_lt());
        const GroupDev g = cd.groups[u];
        col[p] = (int32_t)j;
        const double v = group_value<W>(cd, cd.T, g.tb, g.te, k, L);
        if (valf) valf[p] = (float)v; else val[p] = v;
      }
    } else if (stage.cap > 0) {
      stage_hits(stage, (uint32_t)i, (uint32_t)cnt, j, u);
    }
    cnt += __popc(b);
  });
  if (!FILL && (threadIdx.x & 31) == 0) rowcnt[i] = cnt;
}

// The presence bits of the table's keys (zeroed by the caller).
template <int W>
__global__ void __launch_bounds__(256) k_hash_bits(const uint64_t* __restrict__ keys, int64_t n,
                                                   uint32_t* __restrict__ bits) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t k[W];
    load_key<W>(keys, i, k);
    const KeyBits x = key_bits(key_hash<W>(k));
    atomicOr(bits + x.word, 1u << (x.first & 31) | 1u << (x.second & 31));
  }
}

// The count pass with the table's presence bits in shared memory: one block of 32 warps per SM, each
// warp taking the next row when it has done one.  Bound by instruction issue (about 60 a round of 32
// visits).  Measured against the plain count pass: 200,000 states of 48 modes 13.3 -> 6.9 ms (7.7 with
// one presence bit a key), 40,000 of 30 modes 3.7 -> 1.7 ms, 150,001 of 15 modes 3.2 -> 2.35 ms.
constexpr int kFiltThreads = 1024, kFiltWarps = kFiltThreads / 32;
constexpr size_t kFiltSmem = kBitsWords * sizeof(uint32_t) + kFiltWarps * sizeof(WalkScratch<true>) +
                             kBinomElems * sizeof(uint32_t);

template <int W>
__global__ void __launch_bounds__(kFiltThreads, 1) k_hcount_filtered(
    const uint64_t* __restrict__ keys, int64_t row0, int64_t n, KeyLayout L, HashView basis, ConnDev cd,
    const uint4* __restrict__ bits, int32_t* __restrict__ rowcnt, StageView stage,
    unsigned long long* __restrict__ next) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  uint32_t* s_bits = reinterpret_cast<uint32_t*>(s_raw);
  WalkScratch<true>* s_walk = reinterpret_cast<WalkScratch<true>*>(s_bits + kBitsWords);
  uint32_t* s_binom = reinterpret_cast<uint32_t*>(s_walk + kFiltWarps);
  for (int x = threadIdx.x; x < kBitsWords / 4; x += kFiltThreads) reinterpret_cast<uint4*>(s_bits)[x] = bits[x];
  fill_binom(s_binom);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (;;) {
    unsigned long long i = 0;
    if (lane == 0) i = atomicAdd(next, 1ull);
    i = __shfl_sync(0xffffffffu, i, 0);
    if ((int64_t)i >= n) return;
    uint64_t k[W];
    load_key<W>(keys, row0 + (int64_t)i, k);
    int cnt = 0;
    walk_connections<W, true>(cd, basis, k, L, s_walk[threadIdx.x >> 5], s_binom, s_bits,
                              [&](int64_t j, uint32_t u) {
      const unsigned b = __ballot_sync(0xffffffffu, j >= 0);
      if (stage.cap > 0) stage_hits(stage, (uint32_t)i, (uint32_t)cnt, j, u);
      cnt += __popc(b);
    });
    if (lane == 0) rowcnt[i] = cnt;
  }
}

template <int W>
void hcount_filtered_launch(const uint64_t* keys, int64_t row0, int64_t n, KeyLayout L, HashView basis,
                            int64_t nkeys, ConnDev cd, uint32_t* bits, int32_t* rowcnt, StageView stage,
                            unsigned long long* next, cudaStream_t s) {
  cudaFuncSetAttribute(k_hcount_filtered<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFiltSmem);
  note_launch(); k_hash_bits<W><<<grid_for(nkeys, 256), 256, 0, s>>>(basis.keys, nkeys, bits);
  note_launch(); k_hcount_filtered<W><<<148, kFiltThreads, kFiltSmem, s>>>(
      keys, row0, n, L, basis, cd, reinterpret_cast<const uint4*>(bits), rowcnt, stage, next);
}

// The entries from kept batches, one warp per batch: every lane has an element to form and the
// writes are consecutive, where a second walk costs as much as the first (fill of 200,000 states of
// 48 modes 15.0 -> 0.42 ms, of 150,001 of 15 modes 5.8 -> 0.88 ms).  Bound by the L1 tag stage
// (scattered group and term records): one 32-byte load a term and the ladder table in shared memory
// took 2.1 ms to 0.88; sharing the groups' terms evenly among the lanes gave a tenth.
template <int W>
__global__ void __launch_bounds__(256) k_hfill_staged(
    const uint64_t* __restrict__ keys, int64_t row0, KeyLayout L, ConnDev cd, StageView stage,
    int64_t nbatch, const int64_t* __restrict__ rowptr, int32_t* __restrict__ col,
    double* __restrict__ val, float* __restrict__ valf) {
  __shared__ double s_T[kLadder4];
  const double* T = stage_ladder(cd, L, s_T);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t b = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); b < nbatch; b += warps) {
    const uint2 e = stage.pair[b * 32 + lane];
    if (e.x == kNoIndex) continue;
    const uint2 h = stage.batch[b];
    uint64_t k[W];
    load_key<W>(keys, row0 + h.x, k);
    const int2 terms = __ldg(reinterpret_cast<const int2*>(cd.groups + e.y));
    const double v = group_value<W>(cd, T, terms.x, terms.y, k, L);
    const int64_t p = rowptr[h.x] + h.y + lane;
    col[p] = (int32_t)e.x;
    if (valf) valf[p] = (float)v; else val[p] = v;
  }
}

// One thread per state (the terms are the same for all, their loads broadcast).
template <int W>
__global__ void __launch_bounds__(128) k_diag(const uint64_t* __restrict__ keys, int64_t row0, int64_t n,
                                              KeyLayout L, ConnDev cd, double* __restrict__ diag) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t k[W];
  load_key<W>(keys, row0 + i, k);
  diag[i] = diag_value<W>(cd, k, L);
}

template <int W>
void hbuild_count_launch(const uint64_t* keys, int64_t row0, int64_t stride, int64_t n, KeyLayout L,
                         HashView basis, ConnDev cd, int32_t* rowcnt, StageView stage,
                         cudaStream_t s) {
  note_launch(); k_hbuild<W, false><<<(unsigned)((n + kWalkWarps - 1) / kWalkWarps), kWalkThreads, 0, s>>>(
      keys, row0, stride, n, L, basis, cd, rowcnt, stage, nullptr, nullptr, nullptr, nullptr);
}
template <int W>
void hbuild_fill_launch(const uint64_t* keys, int64_t row0, int64_t n, KeyLayout L,
                        HashView basis, ConnDev cd, const int64_t* rowptr, int32_t* col,
                        double* val, float* valf, cudaStream_t s) {
  note_launch(); k_hbuild<W, true><<<(unsigned)((n + kWalkWarps - 1) / kWalkWarps), kWalkThreads, 0, s>>>(
      keys, row0, 1, n, L, basis, cd, nullptr, StageView{}, rowptr, col, val, valf);
}
template <int W>
void hbuild_fill_staged_launch(const uint64_t* keys, int64_t row0, KeyLayout L, ConnDev cd,
                               StageView stage, int64_t nbatch, const int64_t* rowptr, int32_t* col,
                               double* val, float* valf, cudaStream_t s) {
  note_launch(); k_hfill_staged<W><<<grid_for(nbatch * 32, 256, 148 * 24), 256, 0, s>>>(
      keys, row0, L, cd, stage, nbatch, rowptr, col, val, valf);
}
template <int W>
void diag_launch(const uint64_t* keys, int64_t row0, int64_t n, KeyLayout L, ConnDev cd, double* diag,
                 cudaStream_t s) {
  note_launch(); k_diag<W><<<(unsigned)((n + 127) / 128), 128, 0, s>>>(keys, row0, n, L, cd, diag);
}

// Y[:, 0:VEC bq] = (D + H_off) X, FP64 vectors, one warp per row (rowprod.cuh).  The diagonal term
// reads X row xrow0 + i (a rank's row block of a sharded matrix multiplies the gathered whole
// block); accum != 0 adds into Y instead (a later column panel).  Eight gathers in flight per lane at
// five blocks per SM (51 registers): against sixteen at four blocks 0.375 : 0.401 ms at 120,011 rows
// and 0.056 : 0.058 ms at 24,000; sixteen win by 3 % only at 300,000 rows.  One warp per row with no
// loop over rows: the hardware evens out the rows' lengths (0.375 : 0.395 ms against 2368 blocks).
constexpr int kSpmmUnroll = 8, kSpmmUnrollF = 16;

template <int BQ, int VEC, typename VT>
__global__ void __launch_bounds__(256, 5) k_spmm(int64_t n, const int64_t* __restrict__ rowptr,
                                                 const int32_t* __restrict__ col,
                                                 const VT* __restrict__ val,
                                                 const double* __restrict__ diag,
                                                 const double* X, int ldx, int bq,
                                                 double* __restrict__ Y, int ldy, int accum,
                                                 int64_t xrow0) {
  chain_wait();
  const int lane = threadIdx.x & 31, cc = lane % BQ;
  const bool on = cc < bq;
  const int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const int64_t beg = __ldg(rowptr + i), end = __ldg(rowptr + i + 1);
  if (accum && end == beg) return;
  double a[VEC];
  row_product<kSpmmUnroll, BQ, VEC>(beg, end, col, val, X, ldx / VEC, cc, on, a);
  if (!on || lane >= BQ) return;
  double* y = Y + i * ldy + cc * VEC;
  const double* xi = X + (xrow0 + i) * ldx + cc * VEC;
  const double d = diag[i];
  double o[VEC];
#pragma unroll
  for (int c = 0; c < VEC; ++c) o[c] = accum ? y[c] + a[c] : fma(d, xi[c], a[c]);
#pragma unroll
  for (int c = 0; c < VEC; ++c) y[c] = o[c];
}

// Mixed-precision form: the gathered vector block is FP32 (each lane owns four adjacent columns,
// one 16-byte gather), the matrix values FP32, the accumulation FP64, and the diagonal term
// multiplies the FP64 block Xd (row i of the rows held, stride ldd).  A 16-column FP32 block row
// is 64 bytes, half the gathered bytes of the FP64 form.  Measured (16 columns, four rows per warp
// -> one): 120,011 rows 0.391 -> 0.314 ms, 60,011 rows of the 48-mode basis 0.141 -> 0.053 ms.
template <int BQ>
__global__ void __launch_bounds__(256, 4) k_spmm_f32x(int64_t n, const int64_t* __restrict__ rowptr,
                                                   const int32_t* __restrict__ col,
                                                   const float* __restrict__ val,
                                                   const double* __restrict__ diag,
                                                   const float* X, int ldx, int bq,
                                                   const double* Xd, int ldd,
                                                   double* __restrict__ Y, int ldy) {
  chain_wait();
  const int lane = threadIdx.x & 31, cc = lane % BQ;
  const bool on = cc < bq;
  const int64_t stride = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += stride) {
    double a[4], xd[4], d = 0.0;
    const bool put = on && lane < BQ;
    if (put) {  // asked for before the row's gathers
      d = diag[i];
#pragma unroll
      for (int c = 0; c < 4; ++c) xd[c] = Xd[i * ldd + 4 * cc + c];
    }
    row_product<kSpmmUnrollF, BQ, 4>(__ldg(rowptr + i), __ldg(rowptr + i + 1), col, val, X,
                                     ldx / 4, cc, on, a);
    if (!put) continue;
    double* y = Y + i * ldy + 4 * cc;
#pragma unroll
    for (int c = 0; c < 4; ++c) y[c] = fma(d, xd[c], a[c]);
  }
}

// Lanes per row group and columns per lane by the block's width: pairs of columns (16-byte gathers)
// when the width, the strides and the addresses allow, else single columns; the widest launch covers
// 32 columns.  Narrow blocks spread a row's entries over the lanes that columns leave free (one
// column, 120,011 rows: 0.546 -> 0.177 ms; two 0.350 -> 0.208; four 0.339 -> 0.230).
template <typename VT>
void spmm_rows_launch(int64_t n, const int64_t* rowptr, const int32_t* col, const VT* val,
                      const double* diag, const double* X, int ldx, int b, double* Y, int ldy,
                      int accum, int64_t xrow0, cudaStream_t s) {
  const bool pairs = (b % 2 == 0) && (ldx % 2 == 0) && (ldy % 2 == 0) &&
                     (reinterpret_cast<uintptr_t>(X) % 16 == 0) &&
                     (reinterpret_cast<uintptr_t>(Y) % 16 == 0);
  const int64_t gr = (n + 7) / 8;
  for (int c0 = 0; c0 < b; c0 += 32) {
    const int w = std::min(32, b - c0), q = pairs ? w / 2 : w;
    note_launch();
#define VHCI_SPMM(BQ, VEC)                                                                        \
  launch_chained(k_spmm<BQ, VEC, VT>, (unsigned)gr, 256, 0, s, n, rowptr, col, val, diag, X + c0, ldx, q,       \
                                                   Y + c0, ldy, accum, xrow0)
    if (pairs) {
      if (q == 1) VHCI_SPMM(1, 2);
      else if (q == 2) VHCI_SPMM(2, 2);
      else if (q <= 4) VHCI_SPMM(4, 2);
      else if (q <= 8) VHCI_SPMM(8, 2);
      else VHCI_SPMM(16, 2);
    } else {
      if (q == 1) VHCI_SPMM(1, 1);
      else if (q <= 4) VHCI_SPMM(4, 1);
      else if (q <= 8) VHCI_SPMM(8, 1);
      else if (q <= 16) VHCI_SPMM(16, 1);
      else VHCI_SPMM(32, 1);
    }
#undef VHCI_SPMM
  }
}

// Partial sums of the squared residuals, one block per run of rows, threads over the columns, eight
// rows' loads in flight.
__global__ void __launch_bounds__(256) k_resid_part(const double* __restrict__ X,
                                                    const double* __restrict__ HX, int64_t n, int ld,
                                                    int kk, const double* __restrict__ theta,
                                                    double* __restrict__ part) {
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = blockIdx.x * per, hi = min(n, lo + per);
  for (int c = threadIdx.x; c < kk; c += blockDim.x) {
    const double th = theta[c];
    double s = 0.0;
#pragma unroll 8
    for (int64_t i = lo; i < hi; ++i) {
      const double r = HX[i * ld + c] - th * X[i * ld + c];
      s = fma(r, r, s);
    }
    part[(int64_t)blockIdx.x * kk + c] = s;
  }
}

// One warp per column: lane l adds the partial sums l, l + 32, ..., the lanes' sums in a fixed tree (one
// thread per column took 40 us for 592 partial sums).
__global__ void __launch_bounds__(256) k_sum_parts(const double* __restrict__ part, int nblk, int kk,
                                                   double* __restrict__ out, int accumulate) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (c >= kk) return;
  double s = 0.0;
#pragma unroll 4
  for (int b = lane; b < nblk; b += 32) s += part[(int64_t)b * kk + c];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[c] = accumulate ? out[c] + s : s;
}

__global__ void k_copy_cols(const double* src, int lds, double* __restrict__ dst,
                            int ldd, int64_t n, int ncol) {
  chain_wait();
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < n * ncol;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / ncol;
    const int c = (int)(idx % ncol);
    dst[i * ldd + c] = src[i * lds + c];
  }
}

// Transposes between the column-major host layout and the row-major blocks, 32 x 32 tiles through
// shared memory; blockIdx.x walks the long dimension.  Bound by HBM; the host's strided loops took
// 25 ms for 60,000 x 100 and 3 ms each way for 150,001 x 16.
__global__ void __launch_bounds__(256) k_cols_to_rows(const double* __restrict__ src, int64_t n, int w,
                                                      double* __restrict__ dst, int ldd) {
  __shared__ double t[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int64_t i0 = (int64_t)blockIdx.x * 32;
  const int j0 = blockIdx.y * 32;
  for (int j = y; j < 32; j += 8)
    if (i0 + x < n && j0 + j < w) t[j][x] = src[(int64_t)(j0 + j) * n + i0 + x];
  __syncthreads();
  for (int i = y; i < 32; i += 8)
    if (i0 + i < n && j0 + x < w) dst[(i0 + i) * ldd + j0 + x] = t[x][i];
}

__global__ void __launch_bounds__(256) k_rows_to_cols(const double* __restrict__ src, int lds, int64_t n,
                                                      int w, double* __restrict__ dst) {
  __shared__ double t[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int64_t i0 = (int64_t)blockIdx.x * 32;
  const int j0 = blockIdx.y * 32;
  for (int i = y; i < 32; i += 8)
    if (i0 + i < n && j0 + x < w) t[x][i] = src[(i0 + i) * lds + j0 + x];
  __syncthreads();
  for (int j = y; j < 32; j += 8)
    if (i0 + x < n && j0 + j < w) dst[(int64_t)(j0 + j) * n + i0 + x] = t[j][x];
}

__global__ void k_random_rows(int64_t r0, int64_t n, int b, double* __restrict__ out) {
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n * b;
       x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = x / b;
    const uint64_t key = ((uint64_t)(r0 + i) << 6) ^ (uint64_t)(x - i * b);
    const double u1 = ((mix64(2 * key + 0x9E3779B97F4A7C15ull) >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    const double u2 = ((mix64(2 * key + 1 + 0x9E3779B97F4A7C15ull) >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    out[x] = sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
  }
}

template <typename VT>
__global__ void k_dense_from_csr(int64_t n, const int64_t* __restrict__ rowptr,
                                 const int32_t* __restrict__ col, const VT* __restrict__ val,
                                 const double* __restrict__ diag, double* __restrict__ A) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    for (int64_t e = rowptr[i]; e < rowptr[i + 1]; ++e) A[i * n + col[e]] = (double)val[e];
    A[i * n + i] = diag[i];
  }
}

__global__ void k_fill_zero(double* p, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    p[i] = 0.0;
}

}  // namespace

void hbuild_count(const uint64_t* keys, int64_t row0, int64_t stride, int64_t n, KeyLayout L,
                  HashView basis, ConnDev cd, int32_t* rowcnt, StageView stage, cudaStream_t s) {
  if (n <= 0) return;
  VHCI_DISPATCH_W(L.W, hbuild_count_launch, keys, row0, stride, n, L, basis, cd, rowcnt, stage, s);
}

bool hcount_filter_pays(int64_t n, int64_t nkeys) { return n >= 16384 && nkeys <= (1 << (kBitsLog - 1)); }

void hcount_filtered(const uint64_t* keys, int64_t row0, int64_t n, KeyLayout L, HashView basis,
                     int64_t nkeys, ConnDev cd, uint32_t* bits, int32_t* rowcnt, StageView stage,
                     unsigned long long* next, cudaStream_t s) {
  cudaMemsetAsync(bits, 0, kBitsWords * sizeof(uint32_t), s);
  cudaMemsetAsync(next, 0, sizeof(unsigned long long), s);
  VHCI_DISPATCH_W(L.W, hcount_filtered_launch, keys, row0, n, L, basis, nkeys, cd, bits, rowcnt, stage,
                  next, s);
}

void hbuild_fill(const uint64_t* keys, int64_t row0, int64_t n, KeyLayout L, HashView basis,
                 ConnDev cd, const int64_t* rowptr, int32_t* col, double* val, float* valf,
                 cudaStream_t s) {
  if (n <= 0) return;
  VHCI_DISPATCH_W(L.W, hbuild_fill_launch, keys, row0, n, L, basis, cd, rowptr, col, val, valf, s);
}

void hbuild_fill_staged(const uint64_t* keys, int64_t row0, KeyLayout L, ConnDev cd, StageView stage,
                        int64_t nbatch, const int64_t* rowptr, int32_t* col, double* val,
                        float* valf, cudaStream_t s) {
  if (nbatch <= 0) return;
  VHCI_DISPATCH_W(L.W, hbuild_fill_staged_launch, keys, row0, L, cd, stage, nbatch, rowptr, col, val,
                  valf, s);
}

void diag_energies(const uint64_t* keys, int64_t row0, int64_t n, KeyLayout L, ConnDev cd,
                   double* diag, cudaStream_t s) {
  if (n <= 0) return;
  VHCI_DISPATCH_W(L.W, diag_launch, keys, row0, n, L, cd, diag, s);
}

// ---- column panels: the off-diagonal entries regrouped by column range -----------------------
// On request (capi.cu) the product runs once per column panel, so that the rows gathered in one
// pass (one panel of the block) stay L2-resident while H streams once.
// Layout: entries of panel p for row i at [prow[p n + i], prow[p n + i + 1]); within a (panel,
// row) cell entries keep their CSR order, so the product is deterministic.

namespace {

// cnt[p n + i] = entries of row i in column panel p (cnt zeroed by the caller).
__global__ void __launch_bounds__(256) k_panel_count(int64_t n, const int64_t* __restrict__ rowptr,
                                                     const int32_t* __restrict__ col, int64_t cw,
                                                     int32_t* __restrict__ cnt) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
       i += warps) {
    const int64_t beg = rowptr[i], end = rowptr[i + 1];
    for (int64_t e0 = beg; e0 < end; e0 += 32) {
      const int64_t e = e0 + lane;
      const bool v = e < end;
      const int p = v ? (int)(col[e] / cw) : -1;
      const unsigned peers = __match_any_sync(full, p);
      if (v && (peers & lanemask_lt()) == 0) atomicAdd(cnt + (int64_t)p * n + i, __popc(peers));
    }
  }
}

template <typename VT>
__global__ void __launch_bounds__(256) k_panel_fill(int64_t n, const int64_t* __restrict__ rowptr,
                                                    const int32_t* __restrict__ col,
                                                    const VT* __restrict__ val, int64_t cw, int P,
                                                    const int64_t* __restrict__ prow,
                                                    int32_t* __restrict__ pcol,
                                                    VT* __restrict__ pval) {
  __shared__ int s_run[8][kMaxPanels];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int* run = s_run[threadIdx.x >> 5];
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5); i < n;
       i += warps) {
    for (int p = lane; p < P; p += 32) run[p] = 0;
    __syncwarp();
    const int64_t beg = rowptr[i], end = rowptr[i + 1];
    for (int64_t e0 = beg; e0 < end; e0 += 32) {
      const int64_t e = e0 + lane;
      const bool v = e < end;
      const int p = v ? (int)(col[e] / cw) : -1;
      const unsigned peers = __match_any_sync(full, p);
      const unsigned below = peers & lanemask_lt();
      if (v) {
        const int64_t pos = prow[(int64_t)p * n + i] + run[p] + __popc(below);
        pcol[pos] = col[e];
        pval[pos] = val[e];
      }
      __syncwarp();
      if (v && below == 0) run[p] += __popc(peers);
      __syncwarp();
    }
  }
}

}  // namespace

void panel_count(int64_t n, const int64_t* rowptr, const int32_t* col, int64_t cw, int32_t* cnt,
                 cudaStream_t s) {
  if (n <= 0) return;
  note_launch(); k_panel_count<<<grid_for(n * 32, 256, 148 * 8), 256, 0, s>>>(n, rowptr, col, cw, cnt);
}

void panel_fill(int64_t n, const int64_t* rowptr, const int32_t* col, const double* val,
                const float* valf, int64_t cw, int P, const int64_t* prow, int32_t* pcol,
                double* pval, float* pvalf, cudaStream_t s) {
  if (n <= 0) return;
  const int g = grid_for(n * 32, 256, 148 * 8);
  note_launch();
  if (valf) k_panel_fill<float><<<g, 256, 0, s>>>(n, rowptr, col, valf, cw, P, prow, pcol, pvalf);
  else k_panel_fill<double><<<g, 256, 0, s>>>(n, rowptr, col, val, cw, P, prow, pcol, pval);
}

void spmm_panels(int64_t n, int P, const int64_t* prow, const int32_t* pcol, const double* pval,
                 const float* pvalf, const double* diag, const double* X, int ldx, int b,
                 double* Y, int ldy, int64_t xrow0, cudaStream_t s) {
  if (n <= 0 || b <= 0) return;
  for (int p = 0; p < P; ++p) {
    if (pvalf) spmm_rows_launch<float>(n, prow + (int64_t)p * n, pcol, pvalf, diag, X, ldx, b, Y, ldy, p > 0, xrow0, s);
    else spmm_rows_launch<double>(n, prow + (int64_t)p * n, pcol, pval, diag, X, ldx, b, Y, ldy, p > 0, xrow0, s);
  }
}

bool spmm_f32x(int64_t n, const int64_t* rowptr, const int32_t* col, const float* val,
               const double* diag, const float* X, int ldx, int b, const double* Xd, int ldd,
               double* Y, int ldy, cudaStream_t s) {
  if (n <= 0 || b <= 0) return true;
  if (b % 4 || ldx % 4 || reinterpret_cast<uintptr_t>(X) % 16) return false;
  const int BQ = b <= 16 ? 4 : 8;  // lanes per row; 4 BQ columns per launch
  const int gr = grid_for(n * 32, 256, 148 * 16);
  for (int c0 = 0; c0 < b; c0 += 4 * BQ) {
    const int bq = std::min(BQ, (b - c0) / 4);
    note_launch();
    if (BQ == 8)
      launch_chained(k_spmm_f32x<8>, gr, 256, 0, s, n, rowptr, col, val, diag, X + c0, ldx, bq, Xd + c0, ldd, Y + c0, ldy);
    else
      launch_chained(k_spmm_f32x<4>, gr, 256, 0, s, n, rowptr, col, val, diag, X + c0, ldx, bq, Xd + c0, ldd, Y + c0, ldy);
  }
  return true;
}

// Compact FP32 copy of ncol columns of a row-major FP64 block (rounded to nearest).
__global__ void k_copy_cols_f32(const double* src, int lds, float* __restrict__ dst,
                                int ldd, int64_t n, int ncol) {
  chain_wait();
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < n * ncol;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / ncol;
    const int c = (int)(idx % ncol);
    dst[i * ldd + c] = (float)src[i * lds + c];
  }
}

void copy_cols_f32(const double* src, int lds, float* dst, int ldd, int64_t n, int ncol,
                   cudaStream_t s) {
  if (n <= 0 || ncol <= 0) return;
  note_launch();
  launch_chained(k_copy_cols_f32, grid_for(n * ncol, 256), 256, 0, s, src, lds, dst, ldd, n, ncol);
}

void spmm(int64_t n, const int64_t* rowptr, const int32_t* col, const double* val,
          const float* valf, const double* diag, const double* X, int ldx, int b, double* Y,
          int ldy, int64_t xrow0, cudaStream_t s) {
  if (n <= 0 || b <= 0) return;
  if (valf) spmm_rows_launch<float>(n, rowptr, col, valf, diag, X, ldx, b, Y, ldy, 0, xrow0, s);
  else spmm_rows_launch<double>(n, rowptr, col, val, diag, X, ldx, b, Y, ldy, 0, xrow0, s);
}

int residual_blocks(int64_t n) {
  int64_t b = (n + 63) / 64;
  if (b > 148 * 8) b = 148 * 8;
  if (b < 1) b = 1;
  return (int)b;
}

void residual_norms(const double* X, const double* HX, int64_t n, int ld, int kk,
                    const double* theta, double* part, int nblk, double* rn2, cudaStream_t s) {
  note_launch(); k_resid_part<<<nblk, 256, 0, s>>>(X, HX, n, ld, kk, theta, part);
  note_launch(); k_sum_parts<<<(kk + 7) / 8, 256, 0, s>>>(part, nblk, kk, rn2, 0);
}

void copy_cols(const double* src, int lds, double* dst, int ldd, int64_t n, int ncol,
               cudaStream_t s) {
  if (n <= 0 || ncol <= 0) return;
  note_launch(); launch_chained(k_copy_cols, grid_for(n * ncol, 256), 256, 0, s, src, lds, dst, ldd, n, ncol);
}

void cols_to_rows(const double* src, int64_t n, int w, double* dst, int ldd, cudaStream_t s) {
  if (n <= 0 || w <= 0) return;
  note_launch();
  k_cols_to_rows<<<dim3((unsigned)((n + 31) / 32), (w + 31) / 32), 256, 0, s>>>(src, n, w, dst, ldd);
}

void rows_to_cols(const double* src, int lds, int64_t n, int w, double* dst, cudaStream_t s) {
  if (n <= 0 || w <= 0) return;
  note_launch();
  k_rows_to_cols<<<dim3((unsigned)((n + 31) / 32), (w + 31) / 32), 256, 0, s>>>(src, lds, n, w, dst);
}

void random_rows(int64_t r0, int64_t n, int b, double* out, cudaStream_t s) {
  if (n <= 0 || b <= 0) return;
  note_launch();
  k_random_rows<<<grid_for(n * b, 256), 256, 0, s>>>(r0, n, b, out);
}

void dense_from_csr(int64_t n, const int64_t* rowptr, const int32_t* col, const double* val,
                    const float* valf, const double* diag, double* A, cudaStream_t s) {
  fill_zero(A, n * n, s);
  if (valf) { note_launch(); k_dense_from_csr<float><<<grid_for(n, 128), 128, 0, s>>>(n, rowptr, col, valf, diag, A); }
  else { note_launch(); k_dense_from_csr<double><<<grid_for(n, 128), 128, 0, s>>>(n, rowptr, col, val, diag, A); }
}

void fill_zero(double* p, int64_t n, cudaStream_t s) {
  if (n > 0) { note_launch(); k_fill_zero<<<grid_for(n, 256), 256, 0, s>>>(p, n); }
}

void reduce_parts(const double* part, int nblk, int nopt, double* out_accum, cudaStream_t s) {
  note_launch(); k_sum_parts<<<(nopt + 7) / 8, 256, 0, s>>>(part, nblk, nopt, out_accum, 1);
}

// ---- incremental build: the stored matrix of the first n_old states, extended by the rows of
// the states appended since (H is symmetric to the bit, so the new columns of the old rows are
// the new rows' entries transposed) ----
namespace {

// add[c] += 1 for every new-row entry in an old column c, and the transposed entries' keys
// (c << 32 | entry index) compacted through cnt (their order is fixed by the sort that follows)
__global__ void k_cross_keys(const int32_t* __restrict__ col, int64_t nnz, int64_t n_old,
                             int32_t* __restrict__ add, uint64_t* __restrict__ keys,
                             unsigned long long* __restrict__ cnt) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < nnz;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int32_t c = col[e];
    if (c < n_old) {
      atomicAdd(add + c, 1);
      keys[atomicAdd(cnt, 1ull)] = ((uint64_t)(uint32_t)c << 32) | (uint64_t)e;
    }
  }
}

// entry -> row of the new rows' CSR (one warp per row)
__global__ void k_entry_rows(const int64_t* __restrict__ rp, int64_t nrows, int32_t* __restrict__ erow) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows;
       r += ((int64_t)gridDim.x * blockDim.x) >> 5)
    for (int64_t e = rp[r] + lane; e < rp[r + 1]; e += 32) erow[e] = (int32_t)r;
}

// merged row lengths: old rows keep their entries and gain add[i]; new rows as built
__global__ void k_merge_len(const int64_t* __restrict__ rp_old, const int32_t* __restrict__ add,
                            const int64_t* __restrict__ rp_new, int64_t n_old, int64_t nn,
                            int32_t* __restrict__ len) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_old + nn;
       i += (int64_t)gridDim.x * blockDim.x)
    len[i] = i < n_old ? (int32_t)(rp_old[i + 1] - rp_old[i]) + add[i]
                       : (int32_t)(rp_new[i - n_old + 1] - rp_new[i - n_old]);
}

// rows [rs[i], rs[i+1]) copied to rd[i].. (one warp per row)
template <typename VT>
__global__ void k_copy_rows(const int64_t* __restrict__ rs, const int32_t* __restrict__ cs,
                            const VT* __restrict__ vs, int64_t nrows, const int64_t* __restrict__ rd,
                            int32_t* __restrict__ cd, VT* __restrict__ vd) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows;
       r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int64_t b = rs[r], m = rs[r + 1] - b, d = rd[r];
    for (int64_t t = lane; t < m; t += 32) {
      cd[d + t] = cs[b + t];
      vd[d + t] = vs[b + t];
    }
  }
}

// the sorted transposed entries to the tails of the old rows: key t of column c goes to position
// rp_all[c] + (old length of c) + (t - first key of c), as column n_old + (its new row)
template <typename VT>
__global__ void k_cross_scatter(const uint64_t* __restrict__ keys, int64_t ncross,
                                const int64_t* __restrict__ xoff, const int64_t* __restrict__ rp_old,
                                const int64_t* __restrict__ rp_all, const int32_t* __restrict__ erow,
                                const VT* __restrict__ vnew, int64_t n_old, int32_t* __restrict__ cd,
                                VT* __restrict__ vd) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ncross;
       t += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[t];
    const int64_t c = (int64_t)(k >> 32), e = (int64_t)(k & 0xffffffffull);
    const int64_t pos = rp_all[c] + (rp_old[c + 1] - rp_old[c]) + (t - xoff[c]);
    cd[pos] = (int32_t)(n_old + erow[e]);
    vd[pos] = vnew[e];
  }
}

}  // namespace

void hmerge_cross_keys(const int32_t* col_new, int64_t nnz_new, int64_t n_old, int32_t* add,
                       uint64_t* keys, unsigned long long* cnt, cudaStream_t s) {
  if (nnz_new <= 0) return;
  note_launch();
  k_cross_keys<<<grid_for(nnz_new, 256, 148 * 8), 256, 0, s>>>(col_new, nnz_new, n_old, add, keys, cnt);
}

void hmerge_entry_rows(const int64_t* rp_new, int64_t nn, int32_t* erow, cudaStream_t s) {
  if (nn <= 0) return;
  note_launch();
  k_entry_rows<<<grid_for(nn * 32, 256, 148 * 8), 256, 0, s>>>(rp_new, nn, erow);
}

void hmerge_lengths(const int64_t* rp_old, const int32_t* add, const int64_t* rp_new, int64_t n_old,
                    int64_t nn, int32_t* len, cudaStream_t s) {
  note_launch();
  k_merge_len<<<grid_for(n_old + nn, 256, 148 * 8), 256, 0, s>>>(rp_old, add, rp_new, n_old, nn, len);
}

void hmerge_copy_rows(const int64_t* rs, const int32_t* cs, const double* vs, const float* vsf,
                      int64_t nrows, const int64_t* rd, int32_t* cd, double* vd, float* vdf,
                      cudaStream_t s) {
  if (nrows <= 0) return;
  note_launch();
  const int g = grid_for(nrows * 32, 256, 148 * 8);
  if (vsf) k_copy_rows<float><<<g, 256, 0, s>>>(rs, cs, vsf, nrows, rd, cd, vdf);
  else k_copy_rows<double><<<g, 256, 0, s>>>(rs, cs, vs, nrows, rd, cd, vd);
}

void hmerge_cross_scatter(const uint64_t* keys, int64_t ncross, const int64_t* xoff,
                          const int64_t* rp_old, const int64_t* rp_all, const int32_t* erow,
                          const double* vnew, const float* vnewf, int64_t n_old, int32_t* cd,
                          double* vd, float* vdf, cudaStream_t s) {
  if (ncross <= 0) return;
  note_launch();
  const int g = grid_for(ncross, 256, 148 * 8);
  if (vnewf)
    k_cross_scatter<float><<<g, 256, 0, s>>>(keys, ncross, xoff, rp_old, rp_all, erow, vnewf, n_old, cd, vdf);
  else
    k_cross_scatter<double><<<g, 256, 0, s>>>(keys, ncross, xoff, rp_old, rp_all, erow, vnew, n_old, cd, vd);
}

}  // namespace vhci
