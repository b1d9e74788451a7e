// Internal declarations shared by the CUDA translation units of
// libmetada_gb300.so.  Not part of the C-ABI.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "metada_gb300.h"

struct mg_context {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;
  void* ws = nullptr;  // device workspace, grown on demand
  size_t ws_bytes = 0;
  void* io_ws = nullptr;  // second workspace of the text I/O (the first holds the text)
  size_t io_ws_bytes = 0;
  cudaEvent_t io_done = nullptr;  // its last use
  void* host_stage = nullptr;  // pinned host staging for small read-backs
  size_t host_stage_bytes = 0;
  std::string last_error;
  mg_letkf_stats stats{};
  int64_t io_host_items = 0;  // lines or values the last text I/O call converted on the host
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};  // stage timing
};

namespace mg {

// Hand-written kernel launches on this host thread (CUB scan/sort kernels and
// memsets are not counted).  Contexts are single-threaded, so the count of a
// thread is the count of the contexts it drives.
extern thread_local int64_t g_launches;

int fail(mg_context* ctx, int code, const std::string& msg);
// Device workspace of at least `bytes`; nullptr (with last_error set) on failure.
void* workspace(mg_context* ctx, size_t bytes);
// The text I/O's second workspace: work enqueued on the context's stream from
// here on waits for its last use, on whatever stream that was.  IoUse marks
// that use's end; a block above the size that is kept is freed there.
void* io_workspace(mg_context* ctx, size_t bytes);
void io_release(mg_context* ctx);
struct IoUse {
  mg_context* ctx;
  ~IoUse() { io_release(ctx); }
};
// Pinned host staging of at least `bytes`.
void* host_stage(mg_context* ctx, size_t bytes);

// Carves 256-byte aligned sub-buffers out of one workspace block.
struct Carver {
  char* base = nullptr;
  size_t off = 0;
  template <typename T>
  T* take(size_t count) {
    off = (off + 255) & ~size_t(255);
    T* p = reinterpret_cast<T*>(base + off);
    off += count * sizeof(T);
    return p;
  }
  template <typename T>
  void reserve(size_t count) {
    off = (off + 255) & ~size_t(255);
    off += count * sizeof(T);
  }
};

// Exclusive prefix sum of n int64 counts into offsets[0..n] (offsets[n] =
// total), using `tmp` (scan_temp_bytes(n) bytes of workspace).
size_t scan_temp_bytes(int64_t n);
cudaError_t exclusive_scan(const int64_t* counts, int64_t* offsets, int64_t n, void* tmp,
                           size_t tmp_bytes, cudaStream_t s);

// Internal stages shared between entry points (device pointers).  skip: where
// *skip is not zero, nothing is written.
cudaError_t launch_mean_pert_members(const double* X, int64_t n, int k, int64_t ld, double* mean,
                                     double* Xp64, float* Xp32, int64_t ldp, cudaStream_t s,
                                     const int* skip = nullptr);
cudaError_t launch_to_point_major(const double* X, int64_t n, int k, int64_t ld, double* mean,
                                  double* P64, float* P32, cudaStream_t s);
cudaError_t launch_point_major_to_members(const double* P, int64_t n, int k, double* X,
                                          int64_t ld, cudaStream_t s, const int* skip = nullptr);
// The same stages for members stored as FP32 (FP64 mean of the widened values).
cudaError_t launch_mean_members_f32(const float* X, int64_t n, int k, int64_t ld, double* mean, cudaStream_t s);
cudaError_t launch_to_point_major_f32(const float* X, int64_t n, int k, int64_t ld, double* mean, float* P32,
                                      cudaStream_t s);
cudaError_t launch_point_major_to_members_f32(const float* P, int64_t n, int k, float* X, int64_t ld,
                                              cudaStream_t s);
// Obs-space prior: ym = rowmean(HX), Y' = HX - ym (FP64 and/or FP32 copies),
// d = yo - ym, rinv = 1/rvar.
cudaError_t launch_obs_prior(const double* HX, const double* yo, const double* rvar, int64_t p,
                             int k, double* Y64, float* Y32, double* d, double* rinv,
                             cudaStream_t s);

// Workspace that mg_select_grid takes (from the start of the context's) for npt grid points.
size_t select_grid_bytes(int64_t npt);

// FP64 contractions on the tensor cores by exact splitting, k <= 112
// (mg_fp64gemm.cu).  obs products: nblk partials of [Y'^T R^-1 Y' (k x k),
// Y'^T R^-1 d (k)] and, with eps, Y'^T R^-1 eps (k x k), from H(X) of the raw
// members; the CTAs' sums of squared innovations (dsq_part, may be null); and
// the ensemble mean of X where mean is set (mean_rides_along).  reduce:
// out[e] = sum over partials (out == part allowed).  update: X_i <- mean +
// sum_j (X_j - mean) T_ji in place, member-major.
struct ObsProducts {
  const double* HX;
  const double* eps;  // or null
  const double* yo;
  const double* rvar;
  int64_t p;
  int k, nblk;
  double* part;
  double* dsq_part;
  const double* X;
  int64_t n, ld;
  double* mean;  // or null
};
int obs_blocks(int64_t p, int num_sms);
bool mean_rides_along(int64_t n);
cudaError_t launch_obs_products(const ObsProducts& a, cudaStream_t s);
cudaError_t launch_reduce_parts(const double* part, int nblk, int64_t len, double* out, cudaStream_t s);
cudaError_t launch_update_fp64(double* X, int64_t ld, int64_t n, int k, const double* mean, const double* T,
                               int num_sms, cudaStream_t s);

// The global ETKF's transform with the symmetric square root
// (mg_letkf_hunt.cu): T_ji = out_scale (wa_j + W_ji) from Gb = [G, b],
// A = diag I + G.  ws: hunt_global_bytes(k) of device memory; afterwards
// *hunt_global_info(ws, k) is zero when the system was left to the FP64 Jacobi.
size_t hunt_global_bytes(int k);
const double* hunt_global_info(const void* ws, int k);
cudaError_t launch_hunt_global(const double* Gb, int k, double diag, double out_scale, void* ws, double* T,
                               cudaStream_t s);

// k x k systems by one factorisation (mg_solve.cu).  etkf: from nblk
// partials of [G, b], T_ji = scale (wa_j + W_ji) with A = diag I + G,
// W = sqrt(k-1) chol_L(A^-1); enkf: T = sqrt(rho) (I + A^-1 (b 1^T + F - G)).
// etkf: *status <- 1 when A is not positive definite, else 0; enkf: set to 1
// (not cleared).
int etkf_chol_parts();  // partials that launch_etkf_chol takes
cudaError_t launch_etkf_chol(const double* part, int nblk, int k, double diag, double scale, double* T, int* status,
                             cudaStream_t s);
cudaError_t launch_enkf_chol(const double* G, const double* F, const double* b, int k, double rho, double* T,
                             float* T32, int* status, cudaStream_t s);

// Tensor-core GEMM (tcgen05): C = A B^T + bias, SiLU if act != 0; A (M x K)
// and B (N x K) BF16 row-major, 16-byte aligned, 1 <= N <= 256, K % 8 == 0.
// Writes C32 (FP32) and/or C16 (BF16) with leading dimension ldc; *err is
// set to 1 (not cleared) if a bounded wait gave up.
int tc_gemm_bf16(mg_context* ctx, const __nv_bfloat16* A, const __nv_bfloat16* B, int M, int N, int K,
                 const float* bias, int act, float* C32, __nv_bfloat16* C16, int ldc, int* err);

}  // namespace mg

#define MG_TRY_CUDA(call)                                                                  \
  do {                                                                                     \
    cudaError_t e_ = (call);                                                               \
    if (e_ != cudaSuccess)                                                                 \
      return mg::fail(ctx, MG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

#define MG_COUNT_LAUNCH() (++mg::g_launches)

#define MG_CHECK_ARG(cond, msg)                              \
  do {                                                       \
    if (!(cond)) return mg::fail(ctx, MG_ERR_ARG, (msg));    \
  } while (0)
