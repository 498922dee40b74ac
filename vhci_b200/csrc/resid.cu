// Residual norms of caller-supplied eigenpairs with the context's Hamiltonian:
// rnorm[j] = || H x_j - theta_j x_j ||, the quantity the reference's eigensolver tests against its
// tolerance (Ham.cpp:363).  One fused pass: each warp forms (H x)_i for a panel of up to 32 columns
// (the row product of the SpMM), subtracts theta x_i, squares, and adds into per-block partial sums
// kept in scratch memory; a second kernel sums the partials in a fixed order.
#include <algorithm>
#include <mutex>
#include <vector>

#include "internal.h"
#include "rowprod.cuh"

namespace vhci {

namespace {

// Two blocks of 20 warps per SM (51 registers, the budget of k_spmm): the scratch holds one row of
// partial sums per block, so the blocks are few and wide.
constexpr int kResidThreads = 640, kResidWarps = kResidThreads / 32;
constexpr int kResidBlocks = 148 * 2;  // partial-sum rows (one per block)
constexpr int kResidUnroll = 8;

// One warp per row forms (H x)_i for up to 32 columns (rowprod.cuh) and keeps the running sums of
// the squared residuals; bound by the gathers from L2 as the product is.  Measured against rows
// shared by 8-byte gathers four at a time: 150,001 rows, 51M entries, 200 vectors 27.1 -> 7.9
// ms; 3,001 rows, 10 vectors 93 -> 29 us a call (both kernels).
template <int BQ, int VEC, typename VT>
__global__ void __launch_bounds__(kResidThreads, 2) k_resid_fused(
    int64_t n, const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col,
    const VT* __restrict__ val, const double* __restrict__ diag, const double* __restrict__ X,
    int ldx, int bq, const double* __restrict__ theta, double* __restrict__ part, int ldp) {
  __shared__ double red[kResidWarps][BQ * VEC];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, cc = lane % BQ;
  const bool on = cc < bq;
  double th[VEC], s[VEC];
#pragma unroll
  for (int c = 0; c < VEC; ++c) {
    th[c] = on ? theta[cc * VEC + c] : 0.0;
    s[c] = 0.0;
  }
  for (int64_t i = (int64_t)blockIdx.x * kResidWarps + wid; i < n;
       i += (int64_t)gridDim.x * kResidWarps) {
    double a[VEC];
    row_product<kResidUnroll, BQ, VEC>(__ldg(rowptr + i), __ldg(rowptr + i + 1), col, val, X,
                                       ldx / VEC, cc, on, a);
    if (on && lane < BQ) {
      const double d = diag[i];
#pragma unroll
      for (int c = 0; c < VEC; ++c) {
        const double xi = X[i * ldx + cc * VEC + c];
        const double r = fma(d, xi, a[c]) - th[c] * xi;
        s[c] = fma(r, r, s[c]);
      }
    }
  }
  // block reduction per column, in a fixed order
  if (lane < BQ) {
#pragma unroll
    for (int c = 0; c < VEC; ++c) red[wid][cc * VEC + c] = s[c];
  }
  __syncthreads();
  if (threadIdx.x < VEC * bq) {
    double t = 0.0;
    for (int q = 0; q < kResidWarps; ++q) t += red[q][threadIdx.x];
    part[(int64_t)blockIdx.x * ldp + threadIdx.x] = t;
  }
}

// One warp per column adds the blocks' partial sums (lane l those of blocks l, l + 32, ...) and the
// lanes' sums in a fixed tree (one thread per column took 34 us of a small call).
__global__ void __launch_bounds__(256) k_resid_finish(const double* __restrict__ part, int nblk,
                                                      int ldp, int k, double* __restrict__ rnorm) {
  const int lane = threadIdx.x & 31;
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (c >= k) return;
  double t = 0.0;
#pragma unroll 4
  for (int q = lane; q < nblk; q += 32) t += part[(int64_t)q * ldp + c];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
  if (lane == 0) rnorm[c] = sqrt(t);
}

// Column pairs (16-byte gathers) when the vectors' width and address allow, else single columns.
template <typename VT>
void resid_launch(int64_t n, const int64_t* rowptr, const int32_t* col, const VT* val,
                  const double* diag, const double* X, int ldx, int k, const double* theta,
                  double* part, double* rnorm, cudaStream_t s) {
  const bool pairs = k % 2 == 0 && ldx % 2 == 0 && reinterpret_cast<uintptr_t>(X) % 16 == 0;
  for (int c0 = 0; c0 < k; c0 += 32) {
    const int w = std::min(32, k - c0), q = pairs ? w / 2 : w;
    note_launch();
#define VHCI_RESID(BQ, VEC)                                                                       \
  k_resid_fused<BQ, VEC, VT><<<kResidBlocks, kResidThreads, 0, s>>>(                                \
      n, rowptr, col, val, diag, X + c0, ldx, q, theta + c0, part + c0, k)
    if (pairs) {
      if (q <= 2) VHCI_RESID(2, 2);
      else if (q <= 4) VHCI_RESID(4, 2);
      else if (q <= 8) VHCI_RESID(8, 2);
      else VHCI_RESID(16, 2);
    } else {
      if (q <= 1) VHCI_RESID(1, 1);
      else if (q <= 4) VHCI_RESID(4, 1);
      else if (q <= 8) VHCI_RESID(8, 1);
      else if (q <= 16) VHCI_RESID(16, 1);
      else VHCI_RESID(32, 1);
    }
#undef VHCI_RESID
  }
  note_launch();
  k_resid_finish<<<(k + 7) / 8, 256, 0, s>>>(part, kResidBlocks, k, k, rnorm);
}

}  // namespace

// Residual norms for k device-resident vectors X (n x k row-major, ld = k) with device theta;
// `part` is scratch of resid_scratch_elems(k) doubles.
int64_t resid_scratch_elems(int k) { return (int64_t)kResidBlocks * k; }

void residual_norms_fused(vhci_ctx* c, const double* X, int k, const double* theta, double* part,
                          double* rnorm) {
  if (c->o.precision == 1)
    resid_launch<float>(c->n, c->rowptr.p, c->col.p, c->valf.p, c->diag.p, X, k, k, theta, part,
                        rnorm, c->st);
  else
    resid_launch<double>(c->n, c->rowptr.p, c->col.p, c->val.p, c->diag.p, X, k, k, theta, part,
                         rnorm, c->st);
}

}  // namespace vhci

using namespace vhci;

extern "C" vhci_status vhci_residual_norms(vhci_ctx* c, const double* X, const double* theta,
                                           double* rnorm, int k) {
  if (!c || !X || !theta || !rnorm || k <= 0) return VHCI_E_INPUT;
  if (is_sharded(c)) return fail(c, VHCI_E_STATE, "vhci_residual_norms on a sharded context");
  if (!c->h_valid || c->h_rows) VTRY(build_h(c, true));
  const int64_t n = c->n;
  DBuf<double> dx, dth, part, dr;
  VCK(dx.reserve((size_t)n * k, c->st));
  VCK(dth.reserve(k, c->st));
  VCK(part.reserve(resid_scratch_elems(k), c->st));
  VCK(dr.reserve(k, c->st));
  VTRY(upload_cols(c, X, n, k, dx.p, k));
  VCK(h2d(c, dth.p, theta, k * sizeof(double)));
  residual_norms_fused(c, dx.p, k, dth.p, part.p, dr.p);
  VCK(d2h(c, rnorm, dr.p, k * sizeof(double)));
  VCK(cudaStreamSynchronize(c->st));
  VCK(cudaGetLastError());
  dx.release(c->st);
  dth.release(c->st);
  part.release(c->st);
  dr.release(c->st);
  return VHCI_OK;
}

// ---- residual norms without allocation ------------------------------------------------------
//
// Some callers cannot allocate device memory at the point where they need this check: a serving
// process whose device memory is owned by its own pool, or code that must not trigger the implicit
// device-wide synchronisation of cudaMalloc/cudaFree in the middle of its work.  For them the
// per-block partial sums live in a fixed array in the library's device memory instead of a buffer
// allocated per call.  The array holds kResidBlocks x kNoAllocMaxCols doubles (606 KB) and stays
// resident on every device that loads the library until the process exits.

namespace {

constexpr int kNoAllocMaxCols = 256;
__device__ __align__(256) double g_resid_scratch[kResidBlocks * kNoAllocMaxCols];

std::mutex g_scratch_mu;
double* g_scratch_dev[128] = {nullptr};  // device address of g_resid_scratch per device ordinal

// Restores the calling thread's current device on every return path.
struct DeviceGuard {
  int prev = -1;
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

// True when p is device (or managed) memory that device `dev` can address.  Asks the runtime
// about the pointer; nothing is allocated.
bool device_pointer_on(const void* p, int dev) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();  // clear the (non-sticky) error an unknown pointer may leave
    return false;
  }
  if (a.type == cudaMemoryTypeManaged) return true;
  return a.type == cudaMemoryTypeDevice && a.device == dev;
}

}  // namespace

extern "C" vhci_status vhci_residual_norms_noalloc(vhci_ctx* c, const double* X_dev,
                                                   const double* theta_dev, double* rnorm_dev,
                                                   int k) {
  if (!c || !X_dev || !theta_dev || !rnorm_dev) return VHCI_E_INPUT;
  if (k <= 0 || k > kNoAllocMaxCols)
    return fail(c, VHCI_E_INPUT,
                "vhci_residual_norms_noalloc: k must be between 1 and 256 (the size of its "
                "fixed scratch array)");
  if (!c->h_valid)
    return fail(c, VHCI_E_STATE,
                "vhci_residual_norms_noalloc: the Hamiltonian is not built; call vhci_build_h "
                "first (building it allocates, this call does not)");
  if (c->h_rows)
    return fail(c, VHCI_E_STATE, "vhci_residual_norms_noalloc: the Hamiltonian is sharded");
  const int dev = c->o.device;
  if (dev < 0 || dev >= 128) return fail(c, VHCI_E_CUDA, "device ordinal out of range");
  DeviceGuard guard;
  VCK(cudaGetDevice(&guard.prev));
  VCK(cudaSetDevice(dev));
  if (!device_pointer_on(X_dev, dev) || !device_pointer_on(theta_dev, dev) ||
      !device_pointer_on(rnorm_dev, dev))
    return fail(c, VHCI_E_INPUT,
                "vhci_residual_norms_noalloc: X_dev, theta_dev and rnorm_dev must be device "
                "memory of the context's device");
  double* scratch = nullptr;
  {
    // set-up, once per device with that device current: host code only has a host-side stand-in
    // for the array's name, so the device address is looked up and kept
    std::lock_guard<std::mutex> lk(g_scratch_mu);
    if (!g_scratch_dev[dev]) {
      void* p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_resid_scratch);
      if (e != cudaSuccess) return cuda_fail(c, e, "cudaGetSymbolAddress(g_resid_scratch)");
      g_scratch_dev[dev] = static_cast<double*>(p);
    }
    scratch = g_scratch_dev[dev];
  }
  // every block writes all of its partial sums, so nothing left from an earlier call is read
  residual_norms_fused(c, X_dev, k, theta_dev, scratch, rnorm_dev);
  VCK(cudaGetLastError());
  VCK(cudaStreamSynchronize(c->st));
  return VHCI_OK;
}
