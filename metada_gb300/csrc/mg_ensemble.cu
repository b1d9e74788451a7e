// Ensemble mean / perturbation formation (Ensemble.hpp:105-151) and the
// member-major <-> point-major transposes used by the analyses.
//
// HBM streaming kernels: every byte of the ensemble is read once and every
// output written once; the member loop runs in member order with separately
// rounded adds so that the mean is bit-identical to the reference's
// `mean += m_i` sequence followed by `mean *= 1.0/k`.
#include "mg_fp64.cuh"
#include "mg_internal.h"

namespace {

constexpr int kTile = 32;  // state indices per transpose tile

template <typename TX>
__global__ void __launch_bounds__(256) mean_pert_members_kernel(
    const TX* __restrict__ X, int64_t n, int k, int64_t ld, double inv_k,
    double* __restrict__ mean, double* __restrict__ Xp64, float* __restrict__ Xp32, int64_t ldp,
    const int* __restrict__ skip) {
  const bool keep = skip && *skip;  // read beside the members
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < n; s += stride) {
    double m = 0.0;
    for (int i = 0; i < k; ++i) m = __dadd_rn(m, (double)__ldg(X + (int64_t)i * ld + s));
    m = __dmul_rn(m, inv_k);
    if (keep) return;
    if (mean) mean[s] = m;
    if (Xp64 || Xp32) {
      for (int i = 0; i < k; ++i) {
        const double v = __dsub_rn((double)__ldg(X + (int64_t)i * ld + s), m);
        if (Xp64) Xp64[(int64_t)i * ldp + s] = v;
        if (Xp32) Xp32[(int64_t)i * ldp + s] = (float)v;
      }
    }
  }
}

// Member-major X -> point-major perturbations P[s*k + i] = X_i[s] - mean[s].
// One block per 32 consecutive state indices; tile staged in shared memory so
// both the member rows (input) and the point rows (output) are coalesced.
template <typename TP>
__global__ void __launch_bounds__(256) to_point_major_kernel(const double* __restrict__ X, int64_t n,
                                                             int k, int64_t ld, double inv_k,
                                                             double* __restrict__ mean,
                                                             TP* __restrict__ P) {
  extern __shared__ double tile[];  // [k][kTile + 1]
  __shared__ double smean[kTile];
  const int64_t s0 = (int64_t)blockIdx.x * kTile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i = warp; i < k; i += nw) {
    const int64_t s = s0 + lane;
    tile[i * (kTile + 1) + lane] = (s < n) ? __ldg(X + (int64_t)i * ld + s) : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < kTile) {
    double m = 0.0;
    for (int i = 0; i < k; ++i) m = __dadd_rn(m, tile[i * (kTile + 1) + threadIdx.x]);
    m = __dmul_rn(m, inv_k);
    smean[threadIdx.x] = m;
    const int64_t s = s0 + threadIdx.x;
    if (mean && s < n) mean[s] = m;
  }
  __syncthreads();
  const int total = kTile * k;
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const int j = e / k, i = e - j * k;
    const int64_t s = s0 + j;
    if (s < n) P[s * k + i] = (TP)__dsub_rn(tile[i * (kTile + 1) + j], smean[j]);
  }
}

// Point-major P[s*k + i] -> member-major X_i[s].
__global__ void __launch_bounds__(256) point_major_to_members_kernel(const double* __restrict__ P,
                                                                     int64_t n, int k,
                                                                     double* __restrict__ X,
                                                                     int64_t ld, const int* __restrict__ skip) {
  extern __shared__ double tile[];  // [kTile][k + 1]
  const bool keep = skip && *skip;  // read beside the rows
  const int64_t s0 = (int64_t)blockIdx.x * kTile;
  const int total = kTile * k;
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const int j = e / k, i = e - j * k;
    const int64_t s = s0 + j;
    tile[j * (k + 1) + i] = (s < n) ? __ldg(P + s * k + i) : 0.0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int i = warp; i < k; i += nw) {
    const int64_t s = s0 + lane;
    if (s < n && !keep) X[(int64_t)i * ld + s] = tile[lane * (k + 1) + i];
  }
}

// FP32 members -> FP32 perturbations: T states a block, a thread each for the
// mean (reads coalesced, adds in member order in FP64), the FP32 tile kept in
// shared memory, then a warp per state for the rows.  One FP64 instruction a
// value is left, the mean's add: widening takes integer operations, and
// x - mean is taken against the mean as two floats, with the error of the
// first difference (Knuth's TwoSum), which rounds as the FP64 difference does
// but for ties within 2^-48.  The kernel above, one warp a block for the mean
// and three FP64 instructions a value, took 1.23 ms for 64 members of 2.6M
// states (1.33 GB); this one 0.46 ms.
template <int T>
__global__ void __launch_bounds__(T) to_point_major_f32_kernel(const float* __restrict__ X, int64_t n, int k,
                                                               int64_t ld, double inv_k, double* __restrict__ mean,
                                                               float* __restrict__ P) {
  extern __shared__ float ftile[];  // [k][T + 1]
  __shared__ float smh[T], sml[T];
  const int64_t s0 = (int64_t)blockIdx.x * T;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int64_t s = s0 + t;
  if (s < n) {
    double m = 0.0;
    const float* x = X + s;
    int i = 0;
    for (; i + 8 <= k; i += 8) {
      float v[8];
      bool special = false;
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = __ldg(x + (int64_t)(i + q) * ld);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        ftile[(i + q) * (T + 1) + t] = v[q];
        special |= mg::wide_special(v[q]);
      }
      if (!special) {
#pragma unroll
        for (int q = 0; q < 8; ++q) m = __dadd_rn(m, mg::wide(v[q]));
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) m = __dadd_rn(m, mg::wide_cvt(v[q]));
      }
    }
    for (; i < k; ++i) {
      const float v = __ldg(x + (int64_t)i * ld);
      ftile[i * (T + 1) + t] = v;
      m = __dadd_rn(m, (double)v);
    }
    m = __dmul_rn(m, inv_k);
    if (mean) mean[s] = m;
    const float h = (float)m;
    smh[t] = h;
    sml[t] = (float)__dsub_rn(m, (double)h);
  }
  __syncthreads();
  const int ns = (n - s0 < T) ? (int)(n - s0) : T;
  for (int j = warp; j < ns; j += T / 32) {
    const float h = smh[j], l = sml[j];
    float* p = P + (s0 + j) * k;
    for (int i = lane; i < k; i += 32) {
      const float x = ftile[i * (T + 1) + j];
      const float d = __fsub_rn(x, h), b = __fadd_rn(d, h);
      const float e = __fadd_rn(__fsub_rn(x, b), __fsub_rn(__fsub_rn(b, d), h));  // x - h - d, exact
      const float r = __fadd_rn(d, __fsub_rn(e, l));
      p[i] = fabsf(d) <= 3.402823466e38f ? r : d;  // no low part where the difference is not finite
    }
  }
}

// FP32 rows -> FP32 members: 64 states a block, no conversions (through FP64,
// 0.58 ms for the same ensemble; now 0.26 ms).
__global__ void __launch_bounds__(256) point_major_to_members_f32_kernel(const float* __restrict__ P, int64_t n, int k,
                                                                         int kp, float* __restrict__ X, int64_t ld) {
  extern __shared__ float ftile[];  // [64][kp], kp odd
  const int64_t s0 = (int64_t)blockIdx.x * 64;
  const int ns = (n - s0 < 64) ? (int)(n - s0) : 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 4
  for (int j = warp; j < ns; j += 8) {
    const float* p = P + (s0 + j) * k;
    for (int i = lane; i < k; i += 32) ftile[j * kp + i] = __ldg(p + i);
  }
  __syncthreads();
  for (int i = warp; i < k; i += 8) {
    float* x = X + (int64_t)i * ld + s0;
    if (lane < ns) x[lane] = ftile[lane * kp + i];
    if (lane + 32 < ns) x[lane + 32] = ftile[(lane + 32) * kp + i];
  }
}

inline int grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 152 * 32) b = 152 * 32;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace

namespace mg {

cudaError_t launch_mean_pert_members(const double* X, int64_t n, int k, int64_t ld, double* mean,
                                     double* Xp64, float* Xp32, int64_t ldp, cudaStream_t s, const int* skip) {
  mean_pert_members_kernel<double><<<grid_for(n, 256), 256, 0, s>>>(X, n, k, ld, 1.0 / (double)k, mean,
                                                                   Xp64, Xp32, ldp, skip);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t launch_to_point_major(const double* X, int64_t n, int k, int64_t ld, double* mean,
                                  double* P64, float* P32, cudaStream_t s) {
  const int64_t blocks = (n + kTile - 1) / kTile;
  const size_t smem = (size_t)k * (kTile + 1) * sizeof(double);
  if (P64)
    to_point_major_kernel<double><<<(unsigned)blocks, 256, smem, s>>>(X, n, k, ld, 1.0 / (double)k,
                                                                              mean, P64);
  else
    to_point_major_kernel<float><<<(unsigned)blocks, 256, smem, s>>>(X, n, k, ld, 1.0 / (double)k,
                                                                             mean, P32);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t launch_point_major_to_members(const double* P, int64_t n, int k, double* X, int64_t ld,
                                          cudaStream_t s, const int* skip) {
  const int64_t blocks = (n + kTile - 1) / kTile;
  const size_t smem = (size_t)kTile * (k + 1) * sizeof(double);
  point_major_to_members_kernel<<<(unsigned)blocks, 256, smem, s>>>(P, n, k, X, ld, skip);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

// Members stored as FP32: the mean in FP64 of the widened values (member
// order), FP32 perturbations point-major, and the FP32 write-back.
cudaError_t launch_mean_members_f32(const float* X, int64_t n, int k, int64_t ld, double* mean, cudaStream_t s) {
  mean_pert_members_kernel<float><<<grid_for(n, 256), 256, 0, s>>>(X, n, k, ld, 1.0 / (double)k, mean, nullptr,
                                                                  nullptr, 0, nullptr);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t launch_to_point_major_f32(const float* X, int64_t n, int k, int64_t ld, double* mean, float* P32,
                                      cudaStream_t s) {
  // As many states a block as 48 KB hold (128 up to 90 members, 64 up to
  // the 128 that the analyses take).
  const double inv_k = 1.0 / (double)k;
  if (k <= 90)
    to_point_major_f32_kernel<128><<<(unsigned)((n + 127) / 128), 128, (size_t)k * 129 * sizeof(float), s>>>(
        X, n, k, ld, inv_k, mean, P32);
  else
    to_point_major_f32_kernel<64><<<(unsigned)((n + 63) / 64), 64, (size_t)k * 65 * sizeof(float), s>>>(
        X, n, k, ld, inv_k, mean, P32);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t launch_point_major_to_members_f32(const float* P, int64_t n, int k, float* X, int64_t ld,
                                              cudaStream_t s) {
  const int kp = k | 1;
  point_major_to_members_f32_kernel<<<(unsigned)((n + 63) / 64), 256, (size_t)64 * kp * sizeof(float), s>>>(P, n, k, kp,
                                                                                                          X, ld);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace mg

extern "C" {

int mg_ens_mean(mg_context* ctx, const double* X, int64_t n, int32_t k, int64_t ld,
                double* mean) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(X && mean && n > 0 && k > 0 && ld >= n, "mg_ens_mean: bad arguments");
  MG_TRY_CUDA(mg::launch_mean_pert_members(X, n, k, ld, mean, nullptr, nullptr, 0, ctx->stream));
  return MG_OK;
}

int mg_ens_mean_pert(mg_context* ctx, const double* X, int64_t n, int32_t k, int64_t ld,
                     double* mean, double* Xp, int64_t ldp) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(X && mean && Xp && n > 0 && k > 0 && ld >= n && ldp >= n,
               "mg_ens_mean_pert: bad arguments");
  MG_TRY_CUDA(mg::launch_mean_pert_members(X, n, k, ld, mean, Xp, nullptr, ldp, ctx->stream));
  return MG_OK;
}

}  // extern "C"
