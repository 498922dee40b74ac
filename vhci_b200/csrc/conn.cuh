// Device helpers shared by the Hamiltonian and PT2 kernels: connection-group targets and the
// FC term sums that give Hamiltonian elements.
#pragma once

#include "ops.h"

namespace vhci {

// One term record, read as one 32-byte load (as its own fields it takes four, and the L1 tag stage is
// what the element sums are bound by).
struct TermRegs {
  double fc;
  uint64_t a, b, c;  // bytes 8 .. 31 of TermDev: nk, mode[6], pw[6], dl[6]
  __device__ __forceinline__ int nk() const { return (int)(a & 255u); }
  template <int J> __device__ __forceinline__ int mode() const { return (int)((a >> (8 * (1 + J))) & 255u); }
  template <int J> __device__ __forceinline__ int pw() const {
    return (int)((J == 0 ? a >> 56 : b >> (8 * (J - 1))) & 255u);
  }
  template <int J> __device__ __forceinline__ int dl() const {
    return (int)(int8_t)(J < 3 ? b >> (8 * (5 + J)) : c >> (8 * (J - 3)));
  }
};
__device__ __forceinline__ TermRegs load_term(const TermDev* t) {
  TermRegs r;
  uint64_t fc;
  asm("ld.global.nc.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(fc), "=l"(r.a), "=l"(r.b), "=l"(r.c) : "l"(t));
  r.fc = __longlong_as_double((long long)fc);
  return r;
}

// Sum of a group's terms for ket key k: each term is fc * prod_j T[pw_j][q(mode_j)][dl_j], multiplied
// left to right and summed in table order (the reference's AnharmPot product and Vij sum order).
// Products and sums use explicit round-to-nearest operations so no multiply-add is contracted:
// the results are the same bits as the reference's separate multiplies and adds.  T: the ladder
// table, in global or shared memory.
template <int W>
__device__ __forceinline__ double group_value(const ConnDev& cd, const double* T, int tb, int te,
                                              const uint64_t (&k)[W], const KeyLayout& L) {
  const int qs = L.qmax + 1;
  double v = 0.0;
  for (int t = tb; t < te; ++t) {
    const TermRegs tm = load_term(cd.terms + t);
    const int nk = tm.nk();
    double tv = tm.fc;
    auto factor = [&](int mode, int pw, int dl) {
      const int q = key_q<W>(k, mode, L.mpw, L.bits);
      tv = __dmul_rn(tv, T[(pw * qs + q) * 13 + dl + 6]);
    };
    factor(tm.mode<0>(), tm.pw<0>(), tm.dl<0>());
    if (nk > 1) factor(tm.mode<1>(), tm.pw<1>(), tm.dl<1>());
    if (nk > 2) factor(tm.mode<2>(), tm.pw<2>(), tm.dl<2>());
    if (nk > 3) factor(tm.mode<3>(), tm.pw<3>(), tm.dl<3>());
    if (nk > 4) factor(tm.mode<4>(), tm.pw<4>(), tm.dl<4>());
    if (nk > 5) factor(tm.mode<5>(), tm.pw<5>(), tm.dl<5>());
    v = __dadd_rn(v, tv);
  }
  return v;
}

// The ladder table of 4-bit keys (7 powers, 16 quanta, 13 changes) fits a block's shared memory.
constexpr int kLadder4 = 7 * 16 * 13;
__device__ __forceinline__ const double* stage_ladder(const ConnDev& cd, const KeyLayout& L, double* s) {
  if (L.qmax != 15) return cd.T;
  for (int x = threadIdx.x; x < kLadder4; x += blockDim.x) s[x] = cd.T[x];
  return s;  // the caller synchronises the block
}

// Diagonal element: harmonic energy (Ham.cpp:211-220 operation order) plus the Delta = 0 terms
// in table order (quartic then sextic); equals the reference's fl(E_i + V_ii).
template <int W>
__device__ __forceinline__ double diag_value(const ConnDev& cd, const uint64_t (&k)[W],
                                             const KeyLayout& L) {
  double e = 0.0;
  for (int m = 0; m < cd.nm; ++m) {
    double ej = 0.5;
    ej = __dadd_rn(ej, (double)key_q<W>(k, m, L.mpw, L.bits));
    ej = __dmul_rn(ej, __ldg(cd.freq + m));
    e = __dadd_rn(e, ej);
  }
  const int qs = L.qmax + 1;
  double v = 0.0;
  for (int t = 0; t < cd.ndterms; ++t) {
    const TermDev tm = cd.dterms[t];
    double tv = tm.fc;
    for (int j = 0; j < tm.nk; ++j) {
      const int q = key_q<W>(k, tm.mode[j], L.mpw, L.bits);
      tv = __dmul_rn(tv, __ldg(cd.T + ((int64_t)tm.pw[j] * qs + q) * 13 + 6));
    }
    v = __dadd_rn(v, tv);
  }
  return __dadd_rn(e, v);
}

// Whether a state k can move by group g: every changed mode stays within [0, qmax] (a state outside
// cannot be in a basis stored with this layout).
template <int W>
__device__ __forceinline__ bool group_applies(const GroupDev& g, const uint64_t (&k)[W],
                                              const KeyLayout& L) {
  for (int c = 0; c < g.nchg; ++c) {
    const int q = key_q<W>(k, g.mode[c], L.mpw, L.bits) + g.delta[c];
    if (q < 0 || q > L.qmax) return false;
  }
  return true;
}

// ---- lowered-mode index: visit only the groups a state can move by --------------------------

// Binomial coefficients C(a, r) for a <= 32, r <= 6 at [a * kBinomR + r]; each block copies them to
// shared memory with fill_binom (followed by __syncthreads).
constexpr int kBinomA = 33, kBinomR = 7, kBinomElems = kBinomA * kBinomR;

struct BinomTable {
  uint32_t c[kBinomElems];
};
constexpr BinomTable make_binom() {
  BinomTable t{};
  for (int a = 0; a < kBinomA; ++a)
    for (int r = 0; r < kBinomR; ++r) {
      uint64_t v = 1;  // C(a, i) after step i; exact at every step
      for (int i = 0; i < r; ++i) v = v * (uint64_t)(a > i ? a - i : 0) / (uint64_t)(i + 1);
      t.c[a * kBinomR + r] = (uint32_t)v;
    }
  return t;
}
static __device__ const BinomTable d_binom = make_binom();

__device__ __forceinline__ void fill_binom(uint32_t* binom) {
  for (int t = threadIdx.x; t < kBinomElems; t += blockDim.x) binom[t] = d_binom.c[t];
}

// Segment of the groups lowering the mode set `key` (lowered_key layout): first group, count.
__device__ __forceinline__ void seg_find(const ConnDev& cd, uint64_t key, int& first, int& count) {
  uint32_t h = (uint32_t)mix64(key) & cd.lmask;
  for (uint32_t probe = 0; probe <= cd.lmask; ++probe) {  // load <= 1/2: ends at an empty slot
    const uint64_t k = __ldg(cd.lkey + h);
    if (k == key) {
      first = __ldg(cd.lseg + 2 * h);
      count = __ldg(cd.lseg + 2 * h + 1);
      return;
    }
    if (k == 0) return;
    h = (h + 1) & cd.lmask;
  }
}

// ---- the connection walk ---------------------------------------------------------------------

constexpr int kWalkThreads = 128, kWalkWarps = kWalkThreads / 32;

// Visits in flight per lane and the rings of one warp, in shared memory.  Plain: two probes a lane, a
// ring of possible hits (31 waiting + 64 new).  Filtered: four visits a lane, a ring of the groups
// whose target may be in the table (31 + 128), and of the possible hits (31 + 32).
template <bool FILTER>
struct WalkScratch {
  static constexpr int kIlp = FILTER ? 4 : 2;
  static constexpr unsigned kRing = FILTER ? 64 : 128, kMaybe = FILTER ? 256 : 1;
  uint2 ring[kRing];        // (index found, group)
  int2 seg[32];             // segments of a batch: end in the flattened list, group - position
  uint32_t maybe[kMaybe];   // groups that passed the filter
  uint8_t exc[128];         // excited modes of the state
};

// Calls hit(j, u) for the states of `tab` that state k is connected to, in warp-uniform rounds: in
// every call each lane holds one connected state (its index j in the table, its group u) or j = -1;
// the states come in a fixed order (by lane within a call), so count and fill passes agree.
//
// A group lowering a mode that is not excited in k cannot apply, so with the lowered-mode index only
// the segments of the subsets of k's excited modes (sizes 0..maxl, r-major then colexicographic
// order) are visited; without it, or when the subsets outnumber half the groups, every group is.
// Most visits miss (3,600 groups a state for 350 connected ones on a 15-mode basis, 12,300 for 93 on
// a 48-mode one), so a visit is kept short: the hash of the target is the state's linear hash plus
// the group's constant, one 32-byte sector of slots is compared by fingerprint, and whatever matches
// goes into a ring.  The target key, the bounds of its quanta and the caller's work are done for 32
// ring entries at a time with every lane busy.  (The bounds come last because they rarely fail on a
// match: a target outside them wraps into other modes' fields and is almost never a basis key.)
// Bound by the L1 tag stage (one scattered sector a visit) and the L2 latency behind it.  Measured,
// count pass: 200,000 states of 48 modes 132 -> 13.3 ms (2.5e9 visits), 150,001 of 15 modes 18.3 ->
// 3.2 ms, against visits that checked the bounds first and probed one slot at a time; two probes in
// flight per lane beat four (13.3 : 15.7 ms, fewer registers), one 32-byte load beats a 16-byte one
// over two slots (14.8 ms) or two of them over four (19.2 ms, four in flight).
//
// FILTER: the table's presence bits are in shared memory (sbits).  A visit is then one bit test (a few
// bank conflicts instead of 32 L1 tag cycles), and only what passes is probed, 32 groups at a time
// with every lane busy.
template <int W, bool FILTER = false, class Hit>
__device__ __forceinline__ void walk_connections(const ConnDev& cd, const HashView& tab,
                                                 const uint64_t (&k)[W], const KeyLayout& L,
                                                 WalkScratch<FILTER>& ws, const uint32_t* binom,
                                                 const uint32_t* sbits, Hit&& hit) {
  using WS = WalkScratch<FILTER>;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint64_t hk = hash_lin<W>(k);
  unsigned head = 0, tail = 0;  // ring positions, the same in every lane
  unsigned mhead = 0, mtail = 0;

  // hands on ring entries, 32 at a time (`all`: the rest too)
  auto drain = [&](bool all) {
    __syncwarp();
    while (tail - head >= 32 || (all && tail != head)) {
      const unsigned have = min(32u, tail - head);
      int64_t j = -1;
      uint32_t u = 0;
      if (lane < have) {
        const uint2 r = ws.ring[(head + lane) % WS::kRing];
        u = r.y;
        uint64_t t[W];
#pragma unroll
        for (int w = 0; w < W; ++w) t[w] = k[w] + (uint64_t)__ldg(cd.wdelta + (int64_t)u * W + w);
        // another key of the same fingerprint (about one visit in 2^31): look the target up in full
        j = key_eq<W>(tab.keys, r.x, t) ? (int64_t)r.x : hash_find<W>(tab, t, key_hash<W>(t));
        if (j >= 0 && !group_applies<W>(cd.groups[u], k, L)) j = -1;
      }
      hit(j, u);
      head += have;
    }
    __syncwarp();
  };
  // slots a, b hold the home of a target with linear hash h of group u: what matches goes to the ring
  auto probe = [&](uint64_t h, uint32_t u, const ulonglong2& a, const ulonglong2& b) {
    const uint32_t fp = hash_fp(h);
    uint64_t s = hash_home(h, tab.mask);
    SlotHit r = match_slots(a, b, fp);
    for (uint64_t it = 0; r.more && it <= tab.mask; it += 4) {
      s = (s + 4) & tab.mask;
      ulonglong2 c, d;
      load_slots(tab.slots + s, c, d);
      r = match_slots(c, d, fp);
    }
    const bool on = r.idx != kNoIndex;
    const unsigned m = __ballot_sync(full, on);
    if (on) ws.ring[(tail + __popc(m & lanemask_lt())) % WS::kRing] = make_uint2(r.idx, u);
    tail += __popc(m);
  };
  const ulonglong2 none = make_ulonglong2(kEmptySlot, kEmptySlot);
  // probes the groups that passed the filter, 32 at a time (`all`: the rest too)
  auto probe_maybe = [&](bool all) {
    __syncwarp();
    while (mtail - mhead >= 32 || (all && mtail != mhead)) {
      const unsigned have = min(32u, mtail - mhead);
      uint32_t u = 0;
      uint64_t h = 0;
      ulonglong2 a = none, b = none;
      if (lane < have) {
        u = ws.maybe[(mhead + lane) % WS::kMaybe];
        h = hash_final(hk + __ldg(cd.hdelta + u));
        load_slots(tab.slots + hash_home(h, tab.mask), a, b);
      }
      probe(h, u, a, b);
      mhead += have;
      if (tail - head >= 32) drain(false);
    }
    __syncwarp();
  };
  // visits the flattened list of the segments in ws.seg
  auto visit = [&](int total) {
    constexpr int ILP = WS::kIlp;
    int at = 0;
    int2 sg = ws.seg[0];
    for (int f0 = 0; f0 < total; f0 += 32 * ILP) {
      uint32_t u[ILP];
      uint64_t h[ILP];
#pragma unroll
      for (int t = 0; t < ILP; ++t) {
        const int f = f0 + 32 * t + lane;
        h[t] = 0;
        u[t] = kNoIndex;
        if (f < total) {
          while (f >= sg.x) sg = ws.seg[++at];
          u[t] = (uint32_t)(f + sg.y);
          h[t] = __ldg(cd.hdelta + u[t]);
        }
      }
      if constexpr (FILTER) {
#pragma unroll
        for (int t = 0; t < ILP; ++t) {
          const KeyBits x = key_bits(hash_final(hk + h[t]));
          const uint32_t s = sbits[x.word];
          const bool on = u[t] != kNoIndex && ((s >> (x.first & 31)) & (s >> (x.second & 31)) & 1u);
          const unsigned m = __ballot_sync(full, on);
          if (on) ws.maybe[(mtail + __popc(m & lanemask_lt())) % WS::kMaybe] = u[t];
          mtail += __popc(m);
        }
        if (mtail - mhead >= 32) probe_maybe(false);
      } else {
        ulonglong2 a[ILP], b[ILP];
#pragma unroll
        for (int t = 0; t < ILP; ++t) {
          h[t] = hash_final(hk + h[t]);
          if (u[t] != kNoIndex) load_slots(tab.slots + hash_home(h[t], tab.mask), a[t], b[t]);
          else a[t] = b[t] = none;
        }
#pragma unroll
        for (int t = 0; t < ILP; ++t) probe(h[t], u[t], a[t], b[t]);
        if (tail - head >= 32) drain(false);
      }
    }
  };

  int e = 0;
  int nsub = -1;
  __syncwarp();  // the previous state's readers of the scratch are done
  if (cd.maxl >= 0) {
    for (int m0 = 0; m0 < cd.nm; m0 += 32) {
      const int m = m0 + lane;
      const bool x = m < cd.nm && key_q<W>(k, m, L.mpw, L.bits) > 0;
      const unsigned b = __ballot_sync(full, x);
      if (x) ws.exc[e + __popc(b & lanemask_lt())] = (uint8_t)m;
      e += __popc(b);
    }
    __syncwarp();
    if (e < kBinomA) {
      int64_t ns = 0;
      for (int r = 0; r <= cd.maxl && r <= e; ++r) ns += binom[e * kBinomR + r];
      if (ns <= cd.ngroups / 2) nsub = (int)ns;
    }
  }
  if (nsub < 0) {
    if (lane == 0) ws.seg[0] = make_int2((int)cd.ngroups, 0);
    __syncwarp();
    visit((int)cd.ngroups);
  }
  for (int s0 = 0; s0 < nsub; s0 += 32) {
    const int s = s0 + lane;
    int first = 0, cnt = 0;
    if (s < nsub) {
      int r = 0;
      uint32_t rem = (uint32_t)s;
      while (rem >= binom[e * kBinomR + r]) rem -= binom[e * kBinomR + r++];
      uint64_t key = (uint64_t)(r + 1);
      int hi = e;  // element i = largest c < hi with C(c, i) <= rem (combinatorial number system)
      for (int i = r; i >= 1; --i) {
        int c = hi - 1;
        while (binom[c * kBinomR + i] > rem) --c;
        rem -= binom[c * kBinomR + i];
        key |= (uint64_t)(ws.exc[c] + 1) << (3 + 7 * (i - 1));
        hi = c;
      }
      seg_find(cd, key, first, cnt);
    }
    int incl = cnt;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(full, incl, d);
      if (lane >= d) incl += v;
    }
    const int total = __shfl_sync(full, incl, 31);
    const unsigned some = __ballot_sync(full, cnt > 0);
    if (cnt > 0) ws.seg[__popc(some & lanemask_lt())] = make_int2(incl, first - (incl - cnt));
    __syncwarp();
    visit(total);
    __syncwarp();
  }
  if constexpr (FILTER) probe_maybe(true);
  drain(true);
}

// ---- staged connections ----------------------------------------------------------------------
// The count pass can keep what it finds, so that the fill need not walk again: batches of up to 32
// (state index, group) pairs in any order, each with its row and the row's entries before it.
// Unused places of a batch hold kNoIndex.  A batch beyond the capacity is only counted.
// Called by the whole warp with the hits of one walk round (j < 0: none in this lane).
__device__ __forceinline__ void stage_hits(const StageView& st, uint32_t row, uint32_t off, int64_t j,
                                           uint32_t u) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(full, j >= 0);
  if (m == 0) return;
  unsigned long long b = 0;
  if (lane == 0) b = atomicAdd(st.cursor, 1ull);
  b = __shfl_sync(full, b, 0);
  if ((int64_t)b >= st.cap) return;
  if (lane == 0) st.batch[b] = make_uint2(row, off);
  const unsigned below = j >= 0 ? m : ~m;
  const int at = __popc(below & lanemask_lt()) + (j >= 0 ? 0 : __popc(m));
  st.pair[b * 32 + at] = make_uint2(j >= 0 ? (uint32_t)j : kNoIndex, u);
}

}  // namespace vhci
