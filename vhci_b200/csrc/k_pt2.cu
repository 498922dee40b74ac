// Epstein-Nesbet PT2 kernels (reference: DoPT2, PT2.cpp:16-154).
//
// The reference loops over every (perturber a, variational state i) pair.  Here the connected
// pairs are generated from the variational side: for each state i and connection group u, the
// target a = i + Delta_u is looked up in the perturber hash; hits become entries (a, i, H_ai) of a
// perturber-row CSR (count pass, scan, fill pass).  A fused kernel then forms
// num_a[n] = sum_i H_ai C_in, E_a = H_aa, and sum_a num_a[n]^2 / (E_n - E_a) per block.
#include <climits>

#include "conn.cuh"
#include "ops.h"

namespace vhci {

namespace {

inline int grid_for(int64_t n, int threads, int max_blocks = 148 * 16) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (int)b;
}

__device__ __forceinline__ PtEntry load_entry(const PtEntry* p) {
  const double2 x = __ldg(reinterpret_cast<const double2*>(p));
  return PtEntry{x.x, (int32_t)__double2loint(x.y), 0};
}

constexpr int kEnThreads = 256;
constexpr int kEnBlocks = 148 * 4;

// One warp per variational state: its connected perturbers (conn.cuh, over the perturber table)
// with indices in [a_lo, a_hi), counted per perturber (and all of them kept in `stage` when it has
// room) or written with their matrix elements.
template <int W, bool FILL>
__global__ void __launch_bounds__(kWalkThreads) k_pt2_gen(
    const uint64_t* __restrict__ keys, int64_t n, KeyLayout L, HashView pert, ConnDev cd,
    int64_t a_lo, int64_t a_hi, int32_t* __restrict__ acount, StageView stage,
    unsigned long long* __restrict__ apos, PtEntry* __restrict__ ent) {
  __shared__ uint32_t s_binom[kBinomElems];
  __shared__ WalkScratch<false> s_walk[kWalkWarps];
  fill_binom(s_binom);
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)kWalkWarps + (threadIdx.x >> 5);
  if (i >= n) return;
  uint64_t k[W];
  load_key<W>(keys, i, k);
  walk_connections<W>(cd, pert, k, L, s_walk[threadIdx.x >> 5], s_binom, nullptr, [&](int64_t a, uint32_t u) {
    if (a < a_lo || a >= a_hi) a = -1;
    if (!FILL) {
      if (a >= 0) atomicAdd(acount + (a - a_lo), 1);
      if (stage.cap > 0) stage_hits(stage, (uint32_t)i, 0, a, u);
    } else if (a >= 0) {
      const unsigned long long p = atomicAdd(apos + (a - a_lo), 1ull);
      const GroupDev g = cd.groups[u];
      ent[p] = PtEntry{group_value<W>(cd, cd.T, g.tb, g.te, k, L), (int32_t)i, 0};
    }
  });
}

// The entries of perturbers [a_lo, a_hi) from kept batches, one warp per batch (as k_hfill_staged);
// apos: each perturber's next place.  60,000 states of 15 modes, 66M entries: 13.2 ms by a walk, 2.9 ms
// from the batches with index and value in two arrays, 1.9 ms with both in one 16-byte entry.
// Bound by the scattered atomics and writes.
template <int W>
__global__ void __launch_bounds__(256) k_pt2_fill_staged(
    const uint64_t* __restrict__ keys, KeyLayout L, ConnDev cd, StageView stage, int64_t nbatch,
    int64_t a_lo, int64_t a_hi, unsigned long long* __restrict__ apos, PtEntry* __restrict__ ent) {
  const int64_t b = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= nbatch) return;
  const uint2 e = stage.pair[b * 32 + (threadIdx.x & 31)];
  const int64_t a = e.x;
  if (e.x == kNoIndex || a < a_lo || a >= a_hi) return;
  const unsigned long long p = atomicAdd(apos + (a - a_lo), 1ull);
  const uint32_t i = stage.batch[b].x;
  uint64_t k[W];
  load_key<W>(keys, i, k);
  const int2 terms = __ldg(reinterpret_cast<const int2*>(cd.groups + e.y));
  ent[p] = PtEntry{group_value<W>(cd, cd.T, terms.x, terms.y, k, L), (int32_t)i, 0};
}

template <int W>
void pt2_count_launch(const uint64_t* keys, int64_t n, KeyLayout L, HashView pert, ConnDev cd,
                      int64_t a_lo, int64_t a_hi, int32_t* acount, StageView stage, cudaStream_t s) {
  note_launch(); k_pt2_gen<W, false><<<(unsigned)((n + kWalkWarps - 1) / kWalkWarps), kWalkThreads, 0, s>>>(
      keys, n, L, pert, cd, a_lo, a_hi, acount, stage, nullptr, nullptr);
}
template <int W>
void pt2_fill_launch(const uint64_t* keys, int64_t n, KeyLayout L, HashView pert, ConnDev cd,
                     int64_t a_lo, int64_t a_hi, unsigned long long* apos, PtEntry* ent,
                     cudaStream_t s) {
  note_launch(); k_pt2_gen<W, true><<<(unsigned)((n + kWalkWarps - 1) / kWalkWarps), kWalkThreads, 0, s>>>(
      keys, n, L, pert, cd, a_lo, a_hi, nullptr, StageView{}, apos, ent);
}
template <int W>
void pt2_fill_staged_launch(const uint64_t* keys, KeyLayout L, ConnDev cd, StageView stage,
                            int64_t nbatch, int64_t a_lo, int64_t a_hi, unsigned long long* apos,
                            PtEntry* ent, cudaStream_t s) {
  note_launch(); k_pt2_fill_staged<W><<<(unsigned)((nbatch + 7) / 8), 256, 0, s>>>(
      keys, L, cd, stage, nbatch, a_lo, a_hi, apos, ent);
}

// One warp per perturber row; the perturbers' diagonal elements come from diag_energies (one lane
// forming them here held up its warp: 8.0 -> 4.2 ms on 832k perturbers, 66M entries, 100 columns).
// Lanes own eigenvector columns n = lane + 32 r.  Each warp keeps
// running sums of num^2/(E_n - E_a) over the rows it visits; the block reduces its warps in
// fixed order into part[block][n].
template <int NR>
__global__ void __launch_bounds__(kEnThreads) k_pt2_en(
    const double* __restrict__ ediag, int64_t na, const int64_t* __restrict__ arowptr, const PtEntry* __restrict__ ent,
    const double* __restrict__ X, int ldx, int nopt,
    const double* __restrict__ E, double* __restrict__ part, int ldp) {
  __shared__ double red[kEnThreads / 32][NR * 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  double en[NR], sum[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const int c = lane + 32 * r;
    en[r] = c < nopt ? E[c] : 0.0;
    sum[r] = 0.0;
  }
  for (int64_t a = blockIdx.x * (int64_t)(blockDim.x >> 5) + wid; a < na; a += warps) {
    double num[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) num[r] = 0.0;
    const int64_t beg = arowptr[a], end = arowptr[a + 1];
    for (int64_t e0 = beg; e0 < end; e0 += 32) {
      const int64_t e = e0 + lane;
      int ii = 0;
      double hh = 0.0;
      if (e < end) {
        const PtEntry x = load_entry(ent + e);
        ii = x.i;
        hh = x.v;
      }
      const int m = (int)(end - e0 < 32 ? end - e0 : 32);
#pragma unroll 4
      for (int t = 0; t < m; ++t) {
        const int i = __shfl_sync(0xffffffffu, ii, t);
        const double h = __shfl_sync(0xffffffffu, hh, t);
        const double* xr = X + (int64_t)i * ldx;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const int c = lane + 32 * r;
          if (c < nopt) num[r] = fma(h, __ldg(xr + c), num[r]);
        }
      }
    }
    const double ea = __ldg(ediag + a);
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const int c = lane + 32 * r;
      if (c < nopt) sum[r] += (num[r] * num[r]) / (en[r] - ea);
    }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r) red[wid][lane + 32 * r] = sum[r];
  __syncthreads();
  for (int c = threadIdx.x; c < nopt; c += blockDim.x) {
    double s = 0.0;
    for (int w = 0; w < kEnThreads / 32; ++w) s += red[w][c];
    part[(int64_t)blockIdx.x * ldp + c] = s;
  }
}

// The EN kernel holds NR <= 8 columns per lane, i.e. at most 256 eigenvector columns; wider
// requests (Nstate > 256; the reference has no such limit, PT2.cpp:29-37) run as column tiles of
// 256, each tile writing its own columns of `part` (leading dimension nopt).
constexpr int kEnMaxCols = 8 * 32;

// ---- fixed entry order within perturber rows --------------------------------------------------
// The fill pass takes slots with atomics, so the order of a row's entries (and with it the FP64
// summation order of num_a) would change from run to run.  Each (a, i) pair occurs once per row
// (distinct connection groups move i to distinct targets), so sorting a row by i gives one
// canonical order, and the EN sums become reproducible bit for bit.

constexpr int kSortWarpCap = 256;  // rows up to this length: one warp

// One warp per row of 2..kSortWarpCap entries: every entry's place is the number of smaller i in the
// row (the i are distinct), counted from the row's indices in shared memory, four a read.  That takes
// m^2 / 16 instructions per lane, and no exchanges of the entries: rows of 80 entries on average 3.0
// -> 1.4 ms on 832k rows against a bitonic sort in shared memory.  Longer rows are left to
// k_pt2_sort_long.
__global__ void __launch_bounds__(256) k_pt2_sort_rows(const int64_t* __restrict__ arowptr,
                                                       int64_t nrows, PtEntry* __restrict__ ent) {
  constexpr int NR = kSortWarpCap / 32;
  __shared__ __align__(16) int32_t sk[8][kSortWarpCap];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = blockIdx.x * (int64_t)(blockDim.x >> 5) + wid; r < nrows; r += warps) {
    const int64_t beg = arowptr[r], end = arowptr[r + 1];
    if (end - beg <= 1 || end - beg > kSortWarpCap) continue;
    const int m = (int)(end - beg), nr = (m + 31) / 32;
    double2 x[NR];
    int key[NR], rank[NR];
    __syncwarp();  // the previous row's readers are done
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (q >= nr) break;
      const int t = lane + 32 * q;
      if (t < m) x[q] = reinterpret_cast<const double2*>(ent)[beg + t];
      key[q] = t < m ? __double2loint(x[q].y) : INT_MAX;
      rank[q] = 0;
      sk[wid][t] = key[q];
    }
    __syncwarp();
    for (int c = 0; c < (m + 3) / 4; ++c) {  // past m: INT_MAX, smaller than nothing
      const int4 o = reinterpret_cast<const int4*>(sk[wid])[c];
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        if (q >= nr) break;
        rank[q] += (o.x < key[q]) + (o.y < key[q]) + (o.z < key[q]) + (o.w < key[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) {
      if (q >= nr) break;
      if (lane + 32 * q < m) reinterpret_cast<double2*>(ent)[beg + rank[q]] = x[q];
    }
  }
}

// One block per long row (rows[] lists them): the row is copied to scratch (tmp at the row's offset,
// soff), then every entry goes to position beg + rank, its rank being the number of smaller i in the
// row (the i are distinct).  Cost m^2 / blockDim per row.
__global__ void __launch_bounds__(256) k_pt2_sort_long(const int64_t* __restrict__ arowptr,
                                                       const int64_t* __restrict__ rows,
                                                       const int64_t* __restrict__ soff,
                                                       PtEntry* __restrict__ ent,
                                                       PtEntry* __restrict__ tmp) {
  __shared__ __align__(16) int32_t tile[2048];
  const int64_t r = rows[blockIdx.x];
  const int64_t beg = arowptr[r], m = arowptr[r + 1] - beg;
  PtEntry* tc = tmp + soff[blockIdx.x];
  for (int64_t t = threadIdx.x; t < m; t += blockDim.x) tc[t] = ent[beg + t];
  __syncthreads();
  for (int64_t t0 = 0; t0 < m; t0 += blockDim.x) {
    const int64_t t = t0 + threadIdx.x;
    const PtEntry mine = t < m ? tc[t] : PtEntry{0.0, INT_MAX, 0};
    int64_t rank = 0;
    for (int64_t q0 = 0; q0 < m; q0 += 2048) {
      const int qn = (int)(m - q0 < 2048 ? m - q0 : 2048);
      __syncthreads();
      for (int q = threadIdx.x; q < (qn + 3) / 4 * 4; q += blockDim.x) tile[q] = q < qn ? tc[q0 + q].i : INT_MAX;
      __syncthreads();
      int below = 0;
#pragma unroll 4
      for (int q = 0; q < (qn + 3) / 4; ++q) {
        const int4 o = reinterpret_cast<const int4*>(tile)[q];
        below += (o.x < mine.i) + (o.y < mine.i) + (o.z < mine.i) + (o.w < mine.i);
      }
      rank += below;
    }
    if (t < m) ent[beg + rank] = mine;
  }
}

// crow[i] = arow[i] - arow[0], i in [0, nrows]: a chunk's row offsets from the whole range's; apos: a
// copy, where the fill counts up.
__global__ void k_pt2_rebase(const int64_t* __restrict__ arow, int64_t nrows,
                             int64_t* __restrict__ crow, unsigned long long* __restrict__ apos) {
  const int64_t base = arow[0];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= nrows;
       i += (int64_t)gridDim.x * blockDim.x) {
    crow[i] = arow[i] - base;
    apos[i] = (unsigned long long)(arow[i] - base);
  }
}

// Lists the rows of at least minlen entries: rows[q] and a disjoint scratch offset soff[q] of
// the row's length, q from an atomic counter (cnt[0] rows, cnt[1] entries).  The order of the
// list does not matter: each listed row is ordered by its own block.
__global__ void k_pt2_list_long(const int64_t* __restrict__ arowptr, int64_t nrows, int minlen,
                                int64_t* __restrict__ rows, int64_t* __restrict__ soff,
                                unsigned long long* __restrict__ cnt) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t len = arowptr[r + 1] - arowptr[r];
    if (len >= minlen) {
      const unsigned long long q = atomicAdd(cnt, 1ull);
      rows[q] = r;
      soff[q] = (int64_t)atomicAdd(cnt + 1, (unsigned long long)len);
    }
  }
}

}  // namespace

void pt2_rebase_rows(const int64_t* arow, int64_t nrows, int64_t* crow, unsigned long long* apos,
                     cudaStream_t s) {
  note_launch();
  k_pt2_rebase<<<grid_for(nrows + 1, 256, 148 * 8), 256, 0, s>>>(arow, nrows, crow, apos);
}

void pt2_list_long(const int64_t* arowptr, int64_t nrows, int64_t* rows, int64_t* soff,
                   unsigned long long* cnt, cudaStream_t s) {
  if (nrows <= 0) return;
  note_launch();
  k_pt2_list_long<<<grid_for(nrows, 256, 148 * 8), 256, 0, s>>>(arowptr, nrows, kSortWarpCap + 1,
                                                                 rows, soff, cnt);
}

void pt2_sort_rows(const int64_t* arowptr, int64_t nrows, PtEntry* ent, cudaStream_t s) {
  if (nrows <= 0) return;
  note_launch();
  k_pt2_sort_rows<<<grid_for(nrows * 32, 256, 148 * 16), 256, 0, s>>>(arowptr, nrows, ent);
}

int pt2_sort_long_min() { return kSortWarpCap + 1; }

void pt2_sort_long(const int64_t* arowptr, const int64_t* rows, const int64_t* soff, int nlong,
                   PtEntry* ent, PtEntry* tmp, cudaStream_t s) {
  if (nlong <= 0) return;
  note_launch();
  k_pt2_sort_long<<<nlong, 256, 0, s>>>(arowptr, rows, soff, ent, tmp);
}

void pt2_count(const uint64_t* keys, int64_t n, KeyLayout L, HashView pert, ConnDev cd,
               int64_t a_lo, int64_t a_hi, int32_t* acount, StageView stage, cudaStream_t s) {
  if (n <= 0) return;
  VHCI_DISPATCH_W(L.W, pt2_count_launch, keys, n, L, pert, cd, a_lo, a_hi, acount, stage, s);
}

void pt2_fill_staged(const uint64_t* keys, KeyLayout L, ConnDev cd, StageView stage, int64_t nbatch,
                     int64_t a_lo, int64_t a_hi, unsigned long long* apos, PtEntry* ent,
                     cudaStream_t s) {
  if (nbatch <= 0) return;
  VHCI_DISPATCH_W(L.W, pt2_fill_staged_launch, keys, L, cd, stage, nbatch, a_lo, a_hi, apos, ent, s);
}

void pt2_fill(const uint64_t* keys, int64_t n, KeyLayout L, HashView pert, ConnDev cd, int64_t a_lo,
              int64_t a_hi, unsigned long long* apos, PtEntry* ent, cudaStream_t s) {
  if (n <= 0) return;
  VHCI_DISPATCH_W(L.W, pt2_fill_launch, keys, n, L, pert, cd, a_lo, a_hi, apos, ent, s);
}

int pt2_en_blocks() { return kEnBlocks; }

bool pt2_en(const double* ediag, int64_t na, const int64_t* arowptr, const PtEntry* ent, const double* X, int ldx, int nopt, const double* E, double* part,
            cudaStream_t s) {
  if (nopt <= 0) return false;
  for (int c0 = 0; c0 < nopt; c0 += kEnMaxCols) {
    const int nc = nopt - c0 < kEnMaxCols ? nopt - c0 : kEnMaxCols;
    switch ((nc + 31) / 32) {
#define VHCI_EN_CASE(R)                                                                        \
  case R:                                                                                      \
    note_launch();                                                                             \
    k_pt2_en<R><<<kEnBlocks, kEnThreads, 0, s>>>(ediag, na, arowptr, ent, X + c0, ldx,  \
                                                 nc, E + c0, part + c0, nopt);                 \
    break;
      VHCI_EN_CASE(1) VHCI_EN_CASE(2) VHCI_EN_CASE(3) VHCI_EN_CASE(4)
      VHCI_EN_CASE(5) VHCI_EN_CASE(6) VHCI_EN_CASE(7) VHCI_EN_CASE(8)
#undef VHCI_EN_CASE
      default:
        return false;
    }
  }
  return true;
}

}  // namespace vhci
