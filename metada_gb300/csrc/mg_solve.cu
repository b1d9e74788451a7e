// k x k systems of the global analyses with A = D0 + Y'^T R^-1 Y' factored
// once: the reference's ETKF transform (inverse and lower Cholesky factor,
// ETKF.hpp:150-159) and the EnKF gain (EnKF.hpp:190-225 in its k-dimensional
// form).
//
// A = U D U^T from the last index up (U unit upper triangular), eliminating
// right-hand-side columns on the way: they become U^-1 B.  For the ETKF the
// columns are the identity's, and chol_L(A^-1) = U^-T D^-1/2 is their
// transpose scaled (mg_letkf_chol.cu has the algebra): row i of T needs only
// column i.  For the EnKF they are b 1^T + F - G, followed by D^-1 and U^-T.
// One system is a chain of k steps, and one SM runs two FP64 multiply-adds per
// clock, so the columns are spread over CTAs, eight each, every CTA repeats
// the factorisation, and a step is kept short (eliminate).
// 64 x 64 grid, k = 32: 129 us by one CTA (inverse and two factorisations)
// -> 30 us; EnKF, k = 64: 354 -> 118 us.
#include <cmath>

#include "mg_fp64.cuh"
#include "mg_internal.h"

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kCols = 8;        // right-hand-side columns per CTA
constexpr int kLdb = kCols + 1;  // and b
constexpr int kMaxParts = 4;     // partials summed here (more are summed on many SMs first)

// Eliminates columns k-1 .. 0 of the packed lower triangle A (rows of length
// i + 1) with the columns B (k x kLdb) alongside: A's rows become the
// multipliers u_l (l < j) of column j, B <- U^-1 B; d and 1/d by column.
// A warp walks a row of A and of B together.  The chain from pivot to pivot
// (multiply-add, reciprocal, multipliers) is what bounds a step: the first
// warp updates the next pivot's row before anything else and leaves its
// multipliers and a copy of the row, while the others update the rest, so a
// step has one barrier and only one warp runs the reciprocal (a warp's FP64
// instruction holds its scheduler's unit 64 cycles even where every warp
// computes the same).
template <int KMAX>
__device__ bool eliminate(double* A, double* B, double* raw, double* dval, double* dinv, int k) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool ok = true;
  // Row j is final: multipliers, copy, pivot (the first warp).
  auto pivot_row = [&](int j) {
    double* rw = A + j * (j + 1) / 2;
    double d = rw[j];
    if (!mg::pivot_ok(d)) {
      ok = false;
      d = 1.0;
    }
    const double r = mg::recip_fp64(d);
    double* copy = raw + (j & 1) * KMAX;
    __syncwarp();
    for (int x = lane; x < j; x += 32) {
      const double a = rw[x];
      copy[x] = a;
      rw[x] = a * r;
    }
    if (lane == 0) {
      dval[j] = d;
      dinv[j] = r;
    }
  };
  auto update_row = [&](int i, int j) {
    const double u = A[j * (j + 1) / 2 + i];
    const double *src = raw + (j & 1) * KMAX, *bj = B + j * kLdb;
    double *ri = A + i * (i + 1) / 2, *bi = B + i * kLdb;
    for (int x = lane; x < i + 1 + kLdb; x += 32) {
      double* dst = x <= i ? ri + x : bi + (x - i - 1);
      *dst = __fma_rn(-u, x <= i ? src[x] : bj[x - i - 1], *dst);
    }
  };
  if (warp == 0) pivot_row(k - 1);
  __syncthreads();
  for (int j = k - 1; j > 0; --j) {
    if (warp == 0) {
      update_row(j - 1, j);
      __syncwarp();
      pivot_row(j - 1);
    }
    for (int i = j - 1 - warp; i >= 0; i -= kWarps)
      if (i < j - 1) update_row(i, j);
    __syncthreads();
  }
  return __syncthreads_and(ok);
}

__device__ __forceinline__ double sum_parts(const double* part, int nblk, int64_t len, int64_t e) {
  double t = 0.0;
  for (int b = 0; b < nblk; ++b) t += part[(size_t)b * len + e];
  return t;
}

// part: nblk partials of [G (k x k), b (k)].  T[j*k + i] = scale (wa_j + W_ji).
template <int KMAX>
__global__ void __launch_bounds__(kThreads) etkf_chol_kernel(const double* __restrict__ part, int nblk, int k,
                                                             double diag, double scale, double* __restrict__ T,
                                                             int* status) {
  extern __shared__ __align__(16) double A[];
  __shared__ double B[KMAX * kLdb], raw[2 * KMAX], dval[KMAX], dinv[KMAX], cd[KMAX];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t len = (int64_t)k * k + k;
  const int c0 = blockIdx.x * kCols;
  for (int e = tid; e < k * k; e += kThreads) {
    const int i = e / k, j = e - i * k;
    if (j <= i) A[i * (i + 1) / 2 + j] = sum_parts(part, nblk, len, e) + (i == j ? diag : 0.0);
  }
  for (int e = tid; e < k * kLdb; e += kThreads) {
    const int r = e / kLdb, q = e - r * kLdb;
    B[e] = q < kCols ? (r == c0 + q ? 1.0 : 0.0) : sum_parts(part, nblk, len, (int64_t)k * k + r);
  }
  __syncthreads();
  const bool ok = eliminate<KMAX>(A, B, raw, dval, dinv, k);
  if (blockIdx.x == 0 && tid == 0) *status = ok ? 0 : 1;
  const double cw = sqrt((double)(k - 1));
  for (int r = tid; r < k; r += kThreads) cd[r] = cw * rsqrt(dval[r]);
  __syncthreads();
  const int i = c0 + warp;  // one row of T per warp
  if (i >= k) return;
  double wa = 0.0;
  for (int r = lane; r <= i; r += 32) wa = __fma_rn(B[r * kLdb + warp], B[r * kLdb + kCols] * dinv[r], wa);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) wa += __shfl_xor_sync(0xffffffffu, wa, off);
  for (int m = lane; m < k; m += 32)
    T[i * k + m] = scale * (wa + (m <= i ? B[m * kLdb + warp] * cd[m] : 0.0));
}

// G (k x k), F (k x k), b (k).  T = sr (I + A^-1 (b 1^T + F - G)), A = G + (k-1) I.
template <int KMAX>
__global__ void __launch_bounds__(kThreads) enkf_chol_kernel(const double* __restrict__ G,
                                                             const double* __restrict__ F,
                                                             const double* __restrict__ b, int k, double sr,
                                                             double* __restrict__ T, float* __restrict__ T32,
                                                             int* status) {
  extern __shared__ __align__(16) double A[];
  __shared__ double B[KMAX * kLdb], raw[2 * KMAX], dval[KMAX], dinv[KMAX];
  const int tid = threadIdx.x;
  const int c0 = blockIdx.x * kCols;
  for (int e = tid; e < k * k; e += kThreads) {
    const int i = e / k, j = e - i * k;
    if (j <= i) A[i * (i + 1) / 2 + j] = G[e] + (i == j ? (double)(k - 1) : 0.0);
  }
  for (int e = tid; e < k * kLdb; e += kThreads) {
    const int r = e / kLdb, q = e - r * kLdb, c = c0 + q;
    B[e] = (q < kCols && c < k) ? (b[r] + F[r * k + c]) - G[r * k + c] : 0.0;
  }
  __syncthreads();
  const bool ok = eliminate<KMAX>(A, B, raw, dval, dinv, k);
  if (!ok && blockIdx.x == 0 && tid == 0) *status = 1;
  for (int e = tid; e < k * kLdb; e += kThreads) B[e] *= dinv[e / kLdb];
  __syncthreads();
  for (int l = 0; l < k - 1; ++l) {  // U^-T
    for (int e = tid; e < (k - 1 - l) * kCols; e += kThreads) {
      const int i = l + 1 + e / kCols, q = e % kCols;
      B[i * kLdb + q] = __fma_rn(-A[i * (i + 1) / 2 + l], B[l * kLdb + q], B[i * kLdb + q]);
    }
    __syncthreads();
  }
  for (int e = tid; e < k * kCols; e += kThreads) {
    const int i = e / kCols, q = e % kCols, c = c0 + q;
    if (c >= k) continue;
    const double t = sr * ((i == c ? 1.0 : 0.0) + B[i * kLdb + q]);
    T[i * k + c] = t;
    if (T32) T32[i * k + c] = (float)t;
  }
}

template <int KMAX>
cudaError_t run_etkf(const double* part, int nblk, int k, double diag, double scale, double* T, int* status,
                     cudaStream_t s) {
  constexpr size_t smem = sizeof(double) * (KMAX * (KMAX + 1) / 2);
  const cudaError_t e =
      cudaFuncSetAttribute(etkf_chol_kernel<KMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  etkf_chol_kernel<KMAX><<<(k + kCols - 1) / kCols, kThreads, smem, s>>>(part, nblk, k, diag, scale, T, status);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

template <int KMAX>
cudaError_t run_enkf(const double* G, const double* F, const double* b, int k, double rho, double* T, float* T32,
                     int* status, cudaStream_t s) {
  constexpr size_t smem = sizeof(double) * (KMAX * (KMAX + 1) / 2);
  const cudaError_t e =
      cudaFuncSetAttribute(enkf_chol_kernel<KMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  enkf_chol_kernel<KMAX><<<(k + kCols - 1) / kCols, kThreads, smem, s>>>(G, F, b, k, std::sqrt(rho), T, T32, status);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace

namespace mg {

int etkf_chol_parts() { return kMaxParts; }

cudaError_t launch_etkf_chol(const double* part, int nblk, int k, double diag, double scale, double* T, int* status,
                             cudaStream_t s) {
  return k <= 32 ? run_etkf<32>(part, nblk, k, diag, scale, T, status, s)
                 : run_etkf<112>(part, nblk, k, diag, scale, T, status, s);
}

cudaError_t launch_enkf_chol(const double* G, const double* F, const double* b, int k, double rho, double* T,
                             float* T32, int* status, cudaStream_t s) {
  return k <= 32 ? run_enkf<32>(G, F, b, k, rho, T, T32, status, s)
                 : run_enkf<112>(G, F, b, k, rho, T, T32, status, s);
}

}  // namespace mg
