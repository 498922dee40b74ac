// Product of a sparse matrix row with a block of vectors, one warp per row; shared by the
// eigensolver's product (k_ham.cu) and the residual norms (resid.cu).
//
// BQ lanes own VEC adjacent columns each (one gather of up to 16 bytes per lane and entry); the
// warp's 32 / BQ such groups take the row's entries in turns of U and add their sums by shuffles.
// The product is bound by the latency and the rate of the gathers from L2.  One row per warp ends
// the wait for the longest of the several rows a warp held before (rows of 60 to 700 entries) and
// gives short matrices more warps: measured on 15- and 48-mode bases (16 columns, FP64, ms, four
// rows per warp -> one): 24,000 rows, 4.9M entries 0.117 -> 0.056; 60,011 rows, 4.0M entries
// 0.119 -> 0.053; 120,011 rows, 38.6M entries 0.493 -> 0.375; 300,000 rows, 121M entries
// 1.495 -> 1.119 (13.9 TB/s of gathered rows).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace vhci {

template <typename XT, int VEC> struct XVec;
template <> struct XVec<double, 1> { using T = double; };
template <> struct XVec<double, 2> { using T = double2; };
template <> struct XVec<float, 4> { using T = float4; };

__device__ __forceinline__ void fma_cols(double (&a)[1], double v, double x) { a[0] = fma(v, x, a[0]); }
__device__ __forceinline__ void fma_cols(double (&a)[2], double v, double2 x) {
  a[0] = fma(v, x.x, a[0]);
  a[1] = fma(v, x.y, a[1]);
}
__device__ __forceinline__ void fma_cols(double (&a)[4], double v, float4 x) {
  a[0] = fma(v, (double)x.x, a[0]);
  a[1] = fma(v, (double)x.y, a[1]);
  a[2] = fma(v, (double)x.z, a[2]);
  a[3] = fma(v, (double)x.w, a[3]);
}

// Four matrix values as one or two 16-byte loads (p 4-entry aligned).
__device__ __forceinline__ void load_vals4(const double* p, double* v) {
  const double2 a = __ldg(reinterpret_cast<const double2*>(p));
  const double2 b = __ldg(reinterpret_cast<const double2*>(p + 2));
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void load_vals4(const float* p, float* v) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}

// Sum over the entries [beg, end) of one row of val * X[col, this lane's columns] into a; ldv: row
// stride of X in lane vectors, cv: this lane's vector of a row.  The whole warp calls this together;
// with on = false a lane gathers nothing.  Every lane returns the sum over the whole row.  X is read by
// ordinary loads: the kernel before a chained product may write it (chain.cuh).
template <int U, int BQ, int VEC, typename VT, typename XT>
__device__ __forceinline__ void row_product(int64_t beg, int64_t end, const int32_t* __restrict__ col,
                                            const VT* __restrict__ val, const XT* X,
                                            int64_t ldv, int cv, bool on, double (&a)[VEC]) {
  using XV = typename XVec<XT, VEC>::T;
  constexpr int SP = 32 / BQ;
  const int sub = (threadIdx.x & 31) / BQ;
  const XV* Xv = reinterpret_cast<const XV*>(X) + cv;
#pragma unroll
  for (int c = 0; c < VEC; ++c) a[c] = 0.0;
  if (on) {
    auto gx = [&](int j) { return Xv[(int64_t)j * ldv]; };
    // single entries up to 4-entry alignment, whole turns of U, then the rest
    int64_t e0 = (beg + 3) & ~int64_t(3);
    if (e0 > end) e0 = end;
    const int64_t e1 = e0 + (end - e0) / U * U;
    for (int64_t e = beg + sub; e < e0; e += SP) fma_cols(a, (double)__ldg(val + e), gx(__ldg(col + e)));
    for (int64_t e = e0 + sub * U; e < e1; e += SP * U) {
      int j[U];
      VT v[U];
#pragma unroll
      for (int u = 0; u < U; u += 4) {
        const int4 jj = __ldg(reinterpret_cast<const int4*>(col + e + u));
        j[u] = jj.x; j[u + 1] = jj.y; j[u + 2] = jj.z; j[u + 3] = jj.w;
        load_vals4(val + e + u, v + u);
      }
      XV x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = gx(j[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) fma_cols(a, (double)v[u], x[u]);
    }
#pragma unroll 4
    for (int64_t e = e1 + sub; e < end; e += SP) fma_cols(a, (double)__ldg(val + e), gx(__ldg(col + e)));
  }
#pragma unroll
  for (int d = BQ; d < 32; d <<= 1)
#pragma unroll
    for (int c = 0; c < VEC; ++c) a[c] += __shfl_xor_sync(0xffffffffu, a[c], d);
}

}  // namespace vhci
