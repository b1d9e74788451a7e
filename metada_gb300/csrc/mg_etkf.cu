// Global ETKF (ETKF.hpp:100-179).
//
//   1. the ensemble mean (Ensemble.hpp:105-151; the mixed path also its
//      perturbations, member-major);
//   2. obs-space prior ym, Y' = HX - ym, d = yo - ym (ETKF.hpp:128-141) and
//   3. Gram G = Y'^T R^-1 Y' and b = Y'^T R^-1 d by obs ranges, partials
//      summed in a fixed order (deterministic), FP64 by exact splitting on
//      the tensor cores (mg_fp64gemm.cu);
//   4. the k x k system: the reference's inverse + llt by one factorisation
//      (mg_solve.cu), or the symmetric square root (mg_letkf_hunt.cu, FP64
//      Jacobi where that does not apply), into the transform T
//      (T_ji = rho (wa_j + W_ji) for the reference, whose perturbations carry
//      the inflation, ETKF.hpp:125);
//   5. Xa_i = xm + sum_j X'_j T_ji over state tiles (mg_fp64gemm.cu).
// The Gram and the k x k solve are FP64 on both paths; the mixed path stores
// X' in FP32 and runs the O(n k^2) update in FP32.
// The reference never recomputes the ensemble mean after the update
// (ETKF.hpp:190-191); mean_out receives that background mean.
#include <algorithm>
#include <mutex>

#include "mg_dense.cuh"
#include "mg_internal.h"

namespace {

constexpr int kThreads = 256;

// Hunt: the symmetric square root by FP64 Jacobi of the reduced system
// [G, b], unless *solved says that launch_hunt_global has written T.
template <typename TE>
__global__ void __launch_bounds__(kThreads) etkf_solve_kernel(const double* __restrict__ Gb, int k, int flags,
                                                              double rho, double tol, int sweep_cap,
                                                              const double* __restrict__ solved,
                                                              TE* __restrict__ Tout, int* status) {
  if (solved && *solved != 0.0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int kp = k + (k & 1), lda = kp + 1;
  TE* A = reinterpret_cast<TE*>(smem_raw);
  TE* V = A + kp * lda;
  TE* bvec = V + kp * lda;
  TE* wa = bvec + kp;
  TE* lam = wa + kp;
  TE* uvec = lam + kp;
  TE* rot = uvec + kp;
  int* pairbuf = reinterpret_cast<int*>(rot + 2 * kp);
  int* misc = pairbuf + kp;
  const int tid = threadIdx.x;
  const bool compat_infl = flags & MG_INFL_COMPAT;
  // The reference inflates the perturbations (ETKF.hpp:125), so its A keeps
  // (k-1) I; the Hunt form puts 1/rho on the prior term instead.
  const double diag = compat_infl ? (double)(k - 1) : (double)(k - 1) / rho;
  for (int e = tid; e < kp * kp; e += kThreads) {
    const int i = e / kp, j = e % kp;
    double s = 0.0;
    if (i < k && j < k) {
      s = Gb[i * k + j];
      if (i == j) s += diag;
    } else if (i == j) {
      s = 1.0;
    }
    A[i * lda + j] = (TE)s;
  }
  for (int i = tid; i < k; i += kThreads) bvec[i] = (TE)Gb[k * k + i];
  __syncthreads();
  int sweeps = 0;
  // In the reference form the inflation is applied to X' rather than Pa.
  const bool ok = mg::solve_transform<TE, 128, kThreads>(A, V, bvec, wa, lam, uvec, rot, pairbuf, misc, k, kp, lda, false, false, rho, (TE)tol, sweep_cap,
                                          &sweeps);
  const TE scale = compat_infl ? (TE)rho : TE(1);
  for (int e = tid; e < k * k; e += kThreads) {
    const int j = e / k, i = e - j * k;
    Tout[j * k + i] = scale * (wa[j] + A[j * lda + i]);
  }
  if (tid == 0 && !ok) *status = 1;
}

// Mixed path: Xa_i[s] = xm[s] + sum_j X'_j[s] T_ji in FP32 for a tile of 32 state indices.
template <typename TE>
__global__ void __launch_bounds__(kThreads) etkf_update_kernel(const TE* __restrict__ Xp, int64_t ldp,
                                                               const double* __restrict__ mean,
                                                               const double* __restrict__ T, int64_t n,
                                                               int k, double* __restrict__ X,
                                                               int64_t ld) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TE* Ts = reinterpret_cast<TE*>(smem_raw);  // k x k
  TE* Xt = Ts + k * k;                       // 32 x (k + 1)
  const int64_t s0 = (int64_t)blockIdx.x * 32;
  for (int e = threadIdx.x; e < k * k; e += kThreads) Ts[e] = (TE)T[e];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = warp; j < k; j += kThreads / 32) {
    const int64_t s = s0 + lane;
    Xt[lane * (k + 1) + j] = (s < n) ? Xp[(int64_t)j * ldp + s] : TE(0);
  }
  __syncthreads();
  const int64_t s = s0 + lane;
  if (s < n) {
    const double m = mean[s];
    for (int i = warp; i < k; i += kThreads / 32) {
      TE acc = TE(0);
      for (int j = 0; j < k; ++j) acc += Xt[lane * (k + 1) + j] * Ts[j * k + i];
      X[(int64_t)i * ld + s] = m + (double)acc;
    }
  }
}

// Device buffers of one analysis.
struct EtkfBuffers {
  double* mean;   // n
  float* Xp;      // n x k perturbations (mixed path)
  double* part;   // nblk x (k x k + k)
  double* T;      // k x k
  int* status;
  void* hunt;     // hunt_global_bytes(k), or null: the FP64 Jacobi solves every system
  int nblk;
};

// Enqueues the analysis; *status is set when the k x k system fails.
cudaError_t enqueue_etkf(const EtkfBuffers& w, bool mixed, int num_sms, double* X, int64_t n, int k, int64_t ld,
                         const double* HX, const double* yo, const double* rvar, int64_t p, double rho, int flags,
                         cudaStream_t s) {
  const int64_t len = (int64_t)k * k + k;
  cudaError_t e;
  const bool chol = flags & MG_SQRT_CHOLESKY;
  const bool along = !mixed && mg::mean_rides_along(n);
  if (!along && (e = mg::launch_mean_pert_members(X, n, k, ld, w.mean, nullptr, mixed ? w.Xp : nullptr, n, s)) !=
                    cudaSuccess)
    return e;
  const mg::ObsProducts op{HX, nullptr, yo, rvar, p, k, w.nblk, w.part, nullptr, X, n, ld, along ? w.mean : nullptr};
  if ((e = mg::launch_obs_products(op, s)) != cudaSuccess) return e;
  // The Cholesky solve sums a few partials itself; more are summed on many SMs first.
  int nparts = w.nblk;
  if (nparts > (chol ? mg::etkf_chol_parts() : 1)) {
    if ((e = mg::launch_reduce_parts(w.part, nparts, len, w.part, s)) != cudaSuccess) return e;
    nparts = 1;
  }
  if (chol) {
    const bool compat_infl = flags & MG_INFL_COMPAT;
    e = mg::launch_etkf_chol(w.part, nparts, k, compat_infl ? (double)(k - 1) : (double)(k - 1) / rho,
                             compat_infl ? rho : 1.0, w.T, w.status, s);
    if (e != cudaSuccess) return e;
  } else {
    if ((e = cudaMemsetAsync(w.status, 0, sizeof(int), s)) != cudaSuccess) return e;
    if (w.hunt) {
      const bool compat_infl = flags & MG_INFL_COMPAT;
      e = mg::launch_hunt_global(w.part, k, compat_infl ? (double)(k - 1) : (double)(k - 1) / rho,
                                 compat_infl ? rho : 1.0, w.hunt, w.T, s);
      if (e != cudaSuccess) return e;
    }
    const int kp = k + (k & 1);
    const size_t smem = sizeof(double) * (2 * (size_t)kp * (kp + 1) + 6 * (size_t)kp) + sizeof(int) * (kp + 8) + 64;
    if ((e = cudaFuncSetAttribute(etkf_solve_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem)) != cudaSuccess)
      return e;
    etkf_solve_kernel<double><<<1, kThreads, smem, s>>>(w.part, k, flags, rho, 1e-14, 30,
                                                             w.hunt ? mg::hunt_global_info(w.hunt, k) : nullptr, w.T,
                                                             w.status);
    MG_COUNT_LAUNCH();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (!mixed) return mg::launch_update_fp64(X, ld, n, k, w.mean, w.T, num_sms, s);
  const size_t usmem = sizeof(float) * ((size_t)k * k + 32 * (size_t)(k + 1));
  if ((e = cudaFuncSetAttribute(etkf_update_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)usmem)) != cudaSuccess)
    return e;
  etkf_update_kernel<float><<<(unsigned)((n + 31) / 32), kThreads, usmem, s>>>(w.Xp, n, w.mean, w.T, n, k, X, ld);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

int run_etkf(mg_context* ctx, bool mixed, double* X, int64_t n, int k, int64_t ld, const double* HX, const double* yo,
             const double* rvar, int64_t p, double rho, int flags, double* mean_out) {
  EtkfBuffers w{};
  w.nblk = mg::obs_blocks(p, ctx->num_sms);
  mg::Carver cv;
  for (int pass = 0; pass < 2; ++pass) {
    w.mean = mean_out ? mean_out : cv.take<double>(n);
    w.Xp = cv.take<float>(mixed ? (size_t)n * k : 1);
    w.part = cv.take<double>((size_t)w.nblk * k * (k + 1));
    w.T = cv.take<double>((size_t)k * k);
    w.status = cv.take<int>(4);
    w.hunt = (flags & MG_SQRT_CHOLESKY) ? nullptr : cv.take<char>(mg::hunt_global_bytes(k));
    if (pass == 1) break;
    void* ws = mg::workspace(ctx, cv.off);
    if (!ws) return MG_ERR_NOMEM;
    cv = mg::Carver{static_cast<char*>(ws), 0};
  }
  cudaStream_t s = ctx->stream;
  MG_TRY_CUDA(enqueue_etkf(w, mixed, ctx->num_sms, X, n, k, ld, HX, yo, rvar, p, rho, flags, s));
  int* hs = static_cast<int*>(mg::host_stage(ctx, sizeof(int)));  // pinned
  if (!hs) return MG_ERR_NOMEM;
  MG_TRY_CUDA(cudaMemcpyAsync(hs, w.status, sizeof(int), cudaMemcpyDeviceToHost, s));
  MG_TRY_CUDA(cudaStreamSynchronize(s));
  if (*hs) return mg::fail(ctx, MG_ERR_NUMERIC, "mg_etkf: the k x k system was not positive definite");
  return MG_OK;
}

}  // namespace

extern "C" int mg_etkf(mg_context* ctx, double* X, int64_t n, int32_t k, int64_t ld,
                       const double* HX, const double* yo, const double* rvar, int64_t p,
                       double rho, int32_t flags, int32_t precision, double* mean_out) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(X && n > 0 && k >= 2 && ld >= n && p >= 1 && HX && yo && rvar && rho > 0.0,
               "mg_etkf: bad arguments (k must be 2..128, p >= 1)");
  MG_CHECK_ARG(precision == MG_PREC_FP64 || precision == MG_PREC_MIXED, "mg_etkf: bad precision");
  MG_CHECK_ARG(k <= 112, "mg_etkf: k must be <= 112 (FP64 k x k solve in shared memory)");
  return run_etkf(ctx, precision == MG_PREC_MIXED, X, n, k, ld, HX, yo, rvar, p, rho, flags, mean_out);
}

// ---------------------------------------------------------------------------
// Allocation-free global ETKF.
//
// Some callers cannot allocate device memory at the point where they run the
// analysis: real-time loops whose memory budget is fixed at start-up, and
// host frameworks that own every device allocation through their own pool.
// mg_etkf_noalloc serves them: it runs the same kernels as mg_etkf, but its
// scratch lives in one file-scope device array of fixed size, so the call
// itself performs no cudaMalloc/cudaFree and no allocating library call.  It
// ends by copying the status word to the host and synchronising the stream.
// The array is part of this library's module: every GPU that loads the
// library keeps kStaticScratchBytes reserved until the process exits.
// ---------------------------------------------------------------------------
namespace {

constexpr size_t kStaticScratchBytes = size_t(32) << 20;  // 32 MiB
constexpr int kMaxDevices = 64;

static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

struct StaticSetup {
  std::mutex mu;
  void* addr[kMaxDevices] = {};
  int sms[kMaxDevices] = {};
};
StaticSetup& static_setup() {
  static StaticSetup s;
  return s;
}

// Device address of g_static_scratch on the current device (and its SM
// count), looked up once per device.  In host code the array's name is only
// a host-side stand-in, never a device address.
cudaError_t static_scratch_for_current_device(void** addr, int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  StaticSetup& st = static_setup();
  std::lock_guard<std::mutex> lock(st.mu);
  if (!st.addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess) return e;
    int n = 0;
    e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    st.addr[dev] = p;
    st.sms[dev] = n;
  }
  *addr = st.addr[dev];
  *sms = st.sms[dev];
  return cudaSuccess;
}

int run_etkf_static(cudaStream_t s, bool mixed, double* X, int64_t n, int k, int64_t ld, const double* HX,
                    const double* yo, const double* rvar, int64_t p, double rho, int flags, double* mean_out) {
  void* base = nullptr;
  int num_sms = 0;
  if (static_scratch_for_current_device(&base, &num_sms) != cudaSuccess) {
    cudaGetLastError();
    return MG_ERR_CUDA;
  }
  // The sizes that the entry point documents: what fits does not depend on
  // how the kernels divide the work (they keep no Y', and in FP64 no X').
  const int nblk = (int)std::max<int64_t>(1, std::min<int64_t>((p + 255) / 256, 2 * num_sms));
  mg::Carver cv;
  cv.reserve<double>(n);
  cv.reserve<char>((mixed ? sizeof(float) : sizeof(double)) * n * k);
  cv.reserve<double>((size_t)(p + 1) * k);
  cv.reserve<double>(p + 1);
  cv.reserve<double>(p + 1);
  cv.reserve<double>((size_t)nblk * k * k);
  cv.reserve<double>((size_t)nblk * k);
  cv.reserve<double>((size_t)k * k);
  cv.reserve<int>(4);
  if (cv.off > kStaticScratchBytes) return MG_ERR_CAPACITY;
  cv = mg::Carver{static_cast<char*>(base), 0};
  EtkfBuffers w{};
  w.nblk = std::min(nblk, mg::obs_blocks(p, num_sms));
  w.mean = mean_out ? mean_out : cv.take<double>(n);
  w.Xp = cv.take<float>(mixed ? (size_t)n * k : 1);
  w.part = cv.take<double>((size_t)w.nblk * k * (k + 1));
  w.T = cv.take<double>((size_t)k * k);
  w.status = cv.take<int>(4);
  if (!(flags & MG_SQRT_CHOLESKY) && cv.off + 256 + mg::hunt_global_bytes(k) <= kStaticScratchBytes)
    w.hunt = cv.take<char>(mg::hunt_global_bytes(k));
  auto cuda = [](cudaError_t e) { return e == cudaSuccess ? MG_OK : (cudaGetLastError(), MG_ERR_CUDA); };
  int rc, hs = 0;
  if ((rc = cuda(enqueue_etkf(w, mixed, num_sms, X, n, k, ld, HX, yo, rvar, p, rho, flags, s))) != MG_OK) return rc;
  if ((rc = cuda(cudaMemcpyAsync(&hs, w.status, sizeof(int), cudaMemcpyDeviceToHost, s))) != MG_OK) return rc;
  if ((rc = cuda(cudaStreamSynchronize(s))) != MG_OK) return rc;
  return hs ? MG_ERR_NUMERIC : MG_OK;
}

}  // namespace

extern "C" int mg_etkf_noalloc(void* stream, double* X, int64_t n, int32_t k, int64_t ld, const double* HX,
                               const double* yo, const double* rvar, int64_t p, double rho, int32_t flags,
                               int32_t precision, double* mean_out) {
  if (!(X && n > 0 && k >= 2 && k <= 112 && ld >= n && p >= 1 && HX && yo && rvar && rho > 0.0))
    return MG_ERR_ARG;
  if (precision != MG_PREC_FP64 && precision != MG_PREC_MIXED) return MG_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return run_etkf_static(s, precision == MG_PREC_MIXED, X, n, k, ld, HX, yo, rvar, p, rho, flags, mean_out);
}
