// Stochastic EnKF with perturbed observations (EnKF.hpp:139-254) in the
// k-dimensional form.
//
// The reference forms the p x p matrix S = Y'Y'^T/(k-1) + R, inverts it and
// builds the n x p gain K = X'Y'^T S^-1/(k-1).  By the push-through identity
// Y'^T (Y'Y'^T + (k-1) R)^-1 = (Y'^T R^-1 Y' + (k-1) I)^-1 Y'^T R^-1, so with
// A = Y'^T R^-1 Y' + (k-1) I (k x k) the update of member i,
//     xa_i = xm + X'_i + K (yo + eps_i - Yb_i),
// becomes Xa = xm 1^T + X' T with T = I + A^-1 Y'^T R^-1 D and
// D = d 1^T + eps - Y' (yo - Yb_i = d - Y'_i).  Y'^T R^-1 D = b 1^T + F - G
// with G = Y'^T R^-1 Y', F = Y'^T R^-1 eps and b = Y'^T R^-1 d: two Gram
// passes over the obs and one k x k Cholesky solve, no p x p matrix.  X' is
// the inflated perturbation sqrt(rho)(x_i - xm) (applyInflation :322-335),
// Y' comes from the raw members (:168-174).  The analysis mean is recomputed
// at the end (:237).  Diagnostics: ||d|| (:184), background and analysis
// spread (:334, :240-253); the gain's max/min and S's condition number need
// the n x p gain or the p x p S and are not formed.
#include <algorithm>
#include <cmath>

#include "mg_internal.h"
#include "mg_update.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kSpreadBlocks = 152 * 8;

// C = sum_o rinv_o U[o]^T W[o] over this CTA's obs range (U, W: p x k
// row-major); with bout, also b = sum_o rinv_o d_o U[o].  TE is the
// arithmetic type (FP64, or FP32 on the mixed path).
template <typename TE, int KMAX>
__global__ void __launch_bounds__(kThreads) enkf_cross_kernel(const TE* __restrict__ U, const TE* __restrict__ W,
                                                              const TE* __restrict__ rinv,
                                                              const TE* __restrict__ dinn, int64_t p, int k,
                                                              int64_t per_block, TE* __restrict__ Cpart,
                                                              TE* __restrict__ bpart) {
  constexpr int CH = (KMAX >= 128 && sizeof(TE) == 8) ? 16 : 32, R = KMAX / 16;
  __shared__ TE Us[CH * KMAX], Ws[CH * KMAX];
  __shared__ TE sr[CH], sd[CH];
  const int tid = threadIdx.x, ti = tid / 16, tj = tid % 16;
  const int64_t o0 = (int64_t)blockIdx.x * per_block;
  const int64_t o1 = min(p, o0 + per_block);
  TE acc[R][R];
#pragma unroll
  for (int a = 0; a < R; ++a)
#pragma unroll
    for (int b = 0; b < R; ++b) acc[a][b] = TE(0);
  TE bacc = TE(0);
  for (int64_t c0 = o0; c0 < o1; c0 += CH) {
    const int cnt = (int)(o1 - c0 < (int64_t)CH ? o1 - c0 : (int64_t)CH);
    for (int e = tid; e < cnt * KMAX; e += kThreads) {
      const int r = e / KMAX, j = e - r * KMAX;
      Us[e] = (j < k) ? U[(c0 + r) * k + j] : TE(0);
      Ws[e] = (j < k) ? W[(c0 + r) * k + j] : TE(0);
    }
    if (tid < cnt) {
      sr[tid] = rinv[c0 + tid];
      sd[tid] = dinn[c0 + tid];
    }
    __syncthreads();
    for (int r = 0; r < cnt; ++r) {
      const TE w = sr[r];
      TE av[R], bv[R];
#pragma unroll
      for (int a = 0; a < R; ++a) av[a] = Us[r * KMAX + ti + 16 * a] * w;
#pragma unroll
      for (int b = 0; b < R; ++b) bv[b] = Ws[r * KMAX + tj + 16 * b];
#pragma unroll
      for (int a = 0; a < R; ++a)
#pragma unroll
        for (int b = 0; b < R; ++b) acc[a][b] += av[a] * bv[b];
    }
    if (bpart && tid < k)
      for (int r = 0; r < cnt; ++r) bacc += (Us[r * KMAX + tid] * sr[r]) * sd[r];
    __syncthreads();
  }
  TE* C = Cpart + (size_t)blockIdx.x * k * k;
#pragma unroll
  for (int a = 0; a < R; ++a)
#pragma unroll
    for (int b = 0; b < R; ++b) {
      const int i = ti + 16 * a, j = tj + 16 * b;
      if (i < k && j < k) C[i * k + j] = acc[a][b];
    }
  if (bpart && tid < k) bpart[(size_t)blockIdx.x * k + tid] = bacc;
}

// out[e] = sum over the nblk partials of element e (len elements each), in
// block order: one thread per element, so the sums of the k x k partials
// run on many SMs instead of inside the one-CTA solve.
template <typename TE>
__global__ void __launch_bounds__(kThreads) reduce_partials_kernel(const TE* __restrict__ part, int nblk, int64_t len,
                                                                   double* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (e >= len) return;
  double t = 0.0;
  for (int b = 0; b < nblk; ++b) t += (double)part[(size_t)b * len + e];
  out[e] = t;
}

// Mean over the members (member order, as the analyses' other means) and the
// CTA's partial of the sum of squared perturbations, in one pass over X; the
// second read of a state's members comes from cache.
//
// FP64 instructions bound it (64 cycles of a scheduler each), so the squares
// of a state are summed in integers: values and mean in fixed point, to half an
// ulp of the state's largest value, their differences as two 28-bit limbs,
// three 64-bit sums of products (exact for up to 128 members).  One FP64
// instruction a value is left of three.  The truncation stays below the mean's
// own rounding.  States with infinities, NaN or only tiny values take FP64.  64 members of 2.6M
// states: 0.94 -> 0.43 ms (1.33 GB).
constexpr int kFixMembers = 128;

__device__ __noinline__ double spread_fp64(const double* __restrict__ x, int k, int64_t ld, double m) {
  double sq = 0.0;
  for (int i = 0; i < k; ++i) {
    const double d = x[(int64_t)i * ld] - m;
    sq = __fma_rn(d, d, sq);
  }
  return sq;
}

// x 2^(1077 - emax), truncated, for |x| with a biased exponent up to emax.
__device__ __forceinline__ int64_t to_fixed(double x, int emax) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  const uint64_t mant = ((uint64_t)(uint32_t)((hi & 0xfffff) | (e ? 0x100000 : 0)) << 32) | (uint32_t)__double2loint(x);
  const int64_t v = (int64_t)((mant << 2) >> min(emax - e, 63));
  return hi < 0 ? -v : v;
}

__global__ void __launch_bounds__(kThreads) mean_spread_kernel(const double* __restrict__ X, int64_t n, int k,
                                                               int64_t ld, double inv_k, double* __restrict__ mean,
                                                               double* __restrict__ partial) {
  __shared__ double red[kThreads / 32];
  double sq = 0.0;
  for (int64_t s = (int64_t)blockIdx.x * kThreads + threadIdx.x; s < n; s += (int64_t)gridDim.x * kThreads) {
    double m = 0.0;
    int mx = 0;  // the largest magnitude's leading word
#pragma unroll 8
    for (int i = 0; i < k; ++i) {
      const double x = X[(int64_t)i * ld + s];
      mx = max(mx, __double2hiint(x) & 0x7fffffff);
      m = __dadd_rn(m, x);
    }
    m = __dmul_rn(m, inv_k);
    mean[s] = m;
    const int emax = (mx >> 20) + 1;  // the mean may round up a binade
    if (k > kFixMembers || emax < 64 || emax >= 0x7ff - 7) {  // below: the sum of 128 values stays finite
      sq += spread_fp64(X + s, k, ld, m);
      continue;
    }
    const int64_t mf = to_fixed(m, emax);
    uint64_t hh = 0, hl = 0, ll = 0;
#pragma unroll 8
    for (int i = 0; i < k; ++i) {
      const int64_t d = to_fixed(X[(int64_t)i * ld + s], emax) - mf;
      const uint64_t a = (uint64_t)(d < 0 ? -d : d);
      const uint32_t dh = (uint32_t)(a >> 28), dl = (uint32_t)a & 0x0fffffffu;
      hh += (uint64_t)dh * dh;
      hl += (uint64_t)dh * dl;
      ll += (uint64_t)dl * dl;
    }
    // (hh 2^56 + 2 hl 2^28 + ll) in units of 2^(2 (emax - 1077))
    const double t = __fma_rn((double)hh, 72057594037927936.0, __fma_rn((double)hl, 536870912.0, (double)ll));
    const double unit = __hiloint2double((emax - 54) << 20, 0);
    sq += (t * unit) * unit;
  }
  for (int off = 16; off > 0; off >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, off);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) t += red[w];
    partial[blockIdx.x] = t;
  }
}

// *out = sum of nb partials by one CTA: thread t sums t, t + kThreads, ...
// in order, then a fixed-order tree (deterministic).
__global__ void __launch_bounds__(kThreads) sum_partials_kernel(const double* __restrict__ partial, int nb,
                                                                double* __restrict__ out) {
  __shared__ double red[kThreads];
  double t = 0.0;
  for (int b = threadIdx.x; b < nb; b += kThreads) t += partial[b];
  red[threadIdx.x] = t;
  __syncthreads();
  for (int h = kThreads / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

template <typename TE>
int launch_cross(mg_context* ctx, const TE* U, const TE* W, const TE* rinv, const TE* d, int64_t p, int k, int nblk,
                 int64_t per_block, TE* Cpart, TE* bpart) {
  if (k <= 32)
    enkf_cross_kernel<TE, 32><<<nblk, kThreads, 0, ctx->stream>>>(U, W, rinv, d, p, k, per_block, Cpart, bpart);
  else if (k <= 64)
    enkf_cross_kernel<TE, 64><<<nblk, kThreads, 0, ctx->stream>>>(U, W, rinv, d, p, k, per_block, Cpart, bpart);
  else
    enkf_cross_kernel<TE, 128><<<nblk, kThreads, 0, ctx->stream>>>(U, W, rinv, d, p, k, per_block, Cpart, bpart);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  return MG_OK;
}

template <typename TE>
int reduce_partials(mg_context* ctx, const TE* part, int nblk, int64_t len, double* out) {
  reduce_partials_kernel<TE><<<(unsigned)((len + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(part, nblk,
                                                                                                       len, out);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  return MG_OK;
}

// Mean and, when sum is given, the sum of squared perturbations.
int mean_spread(mg_context* ctx, const double* X, int64_t n, int k, int64_t ld, double* mean, double* partial,
                double* sum) {
  cudaStream_t s = ctx->stream;
  if (!sum) {
    MG_TRY_CUDA(mg::launch_mean_pert_members(X, n, k, ld, mean, nullptr, nullptr, 0, s));
    return MG_OK;
  }
  const int nb = (int)std::min<int64_t>((n + kThreads - 1) / kThreads, kSpreadBlocks);
  mean_spread_kernel<<<nb, kThreads, 0, s>>>(X, n, k, ld, 1.0 / (double)k, mean, partial);
  MG_COUNT_LAUNCH();
  sum_partials_kernel<<<1, kThreads, 0, s>>>(partial, nb, sum);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  return MG_OK;
}

int finish(mg_context* ctx, int64_t n, int k, double rho, const double* mean, double* mean_out, const int* status,
           const double* sums, mg_enkf_diag* diag) {
  cudaStream_t s = ctx->stream;
  if (mean_out) MG_TRY_CUDA(cudaMemcpyAsync(mean_out, mean, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
  int hs = 0;
  double hsum[3] = {0.0, 0.0, 0.0};
  MG_TRY_CUDA(cudaMemcpyAsync(&hs, status, sizeof(int), cudaMemcpyDeviceToHost, s));
  if (diag) MG_TRY_CUDA(cudaMemcpyAsync(hsum, sums, sizeof(hsum), cudaMemcpyDeviceToHost, s));
  MG_TRY_CUDA(cudaStreamSynchronize(s));
  if (hs) return mg::fail(ctx, MG_ERR_NUMERIC, "mg_enkf: the k x k system was not positive definite");
  if (diag) {
    const double nk = (double)n * (double)k;
    diag->innovation_norm = std::sqrt(hsum[0]);
    diag->background_spread = std::sqrt(rho * hsum[1] / nk);
    diag->analysis_spread = std::sqrt(hsum[2] / nk);
  }
  return MG_OK;
}

// FP64 path: every stage in FP64 (the contractions by exact splitting on the
// tensor cores), the analysis mean and spread recomputed from the analysed
// members in member order.
int run_enkf_fp64(mg_context* ctx, double* X, int64_t n, int k, int64_t ld, const double* HX, const double* yo,
                  const double* rvar, const double* eps, int64_t p, double rho, double* mean_out,
                  mg_enkf_diag* diag) {
  const int nblk = mg::obs_blocks(p, ctx->num_sms);
  const int64_t kk = (int64_t)k * k;
  mg::Carver cv;
  double *mean = nullptr, *part = nullptr, *T = nullptr, *red = nullptr, *sums = nullptr;
  int* status = nullptr;
  for (int pass = 0; pass < 2; ++pass) {
    mean = cv.take<double>(n);
    part = cv.take<double>((size_t)nblk * (2 * kk + k));
    T = cv.take<double>(kk);
    red = cv.take<double>(std::max(kSpreadBlocks, nblk));
    sums = cv.take<double>(4);
    status = cv.take<int>(4);
    if (pass == 1) break;
    void* ws = mg::workspace(ctx, cv.off);
    if (!ws) return MG_ERR_NOMEM;
    cv = mg::Carver{static_cast<char*>(ws), 0};
  }
  cudaStream_t s = ctx->stream;
  int rc;
  if ((rc = mean_spread(ctx, X, n, k, ld, mean, red, diag ? sums + 1 : nullptr)) != MG_OK) return rc;
  const mg::ObsProducts op{HX, eps, yo, rvar, p, k, nblk, part, diag ? red : nullptr, nullptr, 0, 0, nullptr};
  MG_TRY_CUDA(mg::launch_obs_products(op, s));
  if (diag) {
    sum_partials_kernel<<<1, kThreads, 0, s>>>(red, nblk, sums + 0);
    MG_COUNT_LAUNCH();
    MG_TRY_CUDA(cudaGetLastError());
  }
  if (nblk > 1) MG_TRY_CUDA(mg::launch_reduce_parts(part, nblk, 2 * kk + k, part, s));
  MG_TRY_CUDA(cudaMemsetAsync(status, 0, sizeof(int) * 4, s));
  MG_TRY_CUDA(mg::launch_enkf_chol(part, part + kk + k, part + kk, k, rho, T, nullptr, status, s));
  // X' carries sqrt(rho) in T, whose columns also hold the identity.
  MG_TRY_CUDA(mg::launch_update_fp64(X, ld, n, k, mean, T, ctx->num_sms, s));
  // Analysis mean and perturbations (Ensemble::RecomputeMean/Perturbations).
  if ((rc = mean_spread(ctx, X, n, k, ld, mean, red, diag ? sums + 2 : nullptr)) != MG_OK) return rc;
  return finish(ctx, n, k, rho, mean, mean_out, status, sums, diag);
}

// Mixed path: Y', the perturbations, d and 1/sigma^2 in FP32 from FP32
// pairs of the FP64 inputs (no FP64 instruction per element), FP32 cross
// products, the k x k solve in FP64, and the fused update (mg_update.cuh)
// that also returns the background and analysis spread sums and the
// analysis mean.
constexpr int kObsWarp = 4;
constexpr int kObsBlock = kObsWarp * (kThreads / 32);
constexpr int kUpdItemS = 512;

__global__ void __launch_bounds__(kThreads) enkf_prior_mixed_kernel(const double* __restrict__ HX,
                                                                    const double* __restrict__ yo,
                                                                    const double* __restrict__ rvar,
                                                                    const double* __restrict__ eps, int64_t p, int k,
                                                                    float* __restrict__ Y32, float* __restrict__ E32,
                                                                    float* __restrict__ d32,
                                                                    float* __restrict__ rinv32,
                                                                    double* __restrict__ dsq_part) {
  __shared__ float wsum[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t ob = (int64_t)blockIdx.x * kObsBlock + (int64_t)warp * kObsWarp;
  double hv[kObsWarp][4], ev[kObsWarp][4];
#pragma unroll
  for (int u = 0; u < kObsWarp; ++u)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int64_t o = ob + u;
      const int i = lane + 32 * t;
      const bool in = o < p && i < k;
      hv[u][t] = in ? HX[o * k + i] : 0.0;
      ev[u][t] = in ? eps[o * k + i] : 0.0;
    }
  const float inv_k = 1.0f / (float)k;
  float dsq = 0.0f;
#pragma unroll
  for (int u = 0; u < kObsWarp; ++u) {
    const int64_t o = ob + u;
    float hh[4], hl[4], s1 = 0.0f;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      mg::split_double(hv[u][t], hh[t], hl[t]);
      s1 += hh[t] + hl[t];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s1 += __shfl_xor_sync(0xffffffffu, s1, off);
    const float m1 = s1 * inv_k;
    float pv[4], s2 = 0.0f;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      pv[t] = (lane + 32 * t < k) ? __fadd_rn(__fsub_rn(hh[t], m1), hl[t]) : 0.0f;
      s2 += pv[t];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, off);
    const float m2 = s2 * inv_k;
    if (o < p) {
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int i = lane + 32 * t;
        if (i < k) {
          float eh, el;
          mg::split_double(ev[u][t], eh, el);
          Y32[o * k + i] = pv[t] - m2;
          E32[o * k + i] = __fadd_rn(eh, el);
        }
      }
      if (lane == 0) {
        float yh, yl, vh, vl;
        mg::split_double(yo[o], yh, yl);
        mg::split_double(rvar[o], vh, vl);
        const float dd = __fsub_rn(__fadd_rn(__fsub_rn(yh, m1), yl), m2);
        d32[o] = dd;
        rinv32[o] = 1.0f / __fadd_rn(vh, vl);
        dsq = fmaf(dd, dd, dsq);
      }
    }
  }
  if (lane == 0) wsum[warp] = dsq;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int w = 0; w < kThreads / 32; ++w) t += wsum[w];
    dsq_part[blockIdx.x] = (double)t;
  }
}

__global__ void __launch_bounds__(mg::kUpdThreads, 2) enkf_update_mixed_kernel(double* X, int64_t ld, int64_t n,
                                                                                 int k, const float* __restrict__ T32,
                                                                                 double* mean,
                                                                                 double* __restrict__ bg_part,
                                                                                 double* __restrict__ an_part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float red[2][mg::kUpdThreads / 32];
  const int64_t a = (int64_t)blockIdx.x * kUpdItemS;
  const int64_t b = min(n, a + kUpdItemS);
  float bg = 0.0f, an = 0.0f;
  mg::update_mixed<true>(X, ld, k, a, b, T32, mean, reinterpret_cast<float*>(smem_raw), k, bg, an);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    bg += __shfl_xor_sync(0xffffffffu, bg, off);
    an += __shfl_xor_sync(0xffffffffu, an, off);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    red[0][warp] = bg;
    red[1][warp] = an;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float tb = 0.0f, ta = 0.0f;
    for (int w = 0; w < mg::kUpdThreads / 32; ++w) {
      tb += red[0][w];
      ta += red[1][w];
    }
    bg_part[blockIdx.x] = (double)tb;
    an_part[blockIdx.x] = (double)ta;
  }
}

int run_enkf_mixed(mg_context* ctx, double* X, int64_t n, int k, int64_t ld, const double* HX, const double* yo,
                   const double* rvar, const double* eps, int64_t p, double rho, double* mean_out,
                   mg_enkf_diag* diag) {
  const int nblk = (int)std::max<int64_t>(1, std::min<int64_t>((p + 255) / 256, 2 * ctx->num_sms));
  const int64_t per_block = (p + nblk - 1) / nblk;
  const int64_t kk = (int64_t)k * k;
  const int nprior = (int)((p + kObsBlock - 1) / kObsBlock);
  const int nupd = (int)((n + kUpdItemS - 1) / kUpdItemS);
  mg::Carver cv;
  cv.reserve<double>(n);
  cv.reserve<float>((size_t)p * k);
  cv.reserve<float>((size_t)p * k);
  cv.reserve<float>(p);
  cv.reserve<float>(p);
  cv.reserve<float>((size_t)nblk * kk);
  cv.reserve<float>((size_t)nblk * kk);
  cv.reserve<float>((size_t)nblk * k);
  cv.reserve<double>(2 * kk + k);
  cv.reserve<double>(kk);
  cv.reserve<float>(kk);
  cv.reserve<double>(nprior);
  cv.reserve<double>(nupd);
  cv.reserve<double>(nupd);
  cv.reserve<double>(4);
  cv.reserve<int>(4);
  void* ws = mg::workspace(ctx, cv.off);
  if (!ws) return MG_ERR_NOMEM;
  cv = mg::Carver{static_cast<char*>(ws), 0};
  double* mean = cv.take<double>(n);
  float* Y32 = cv.take<float>((size_t)p * k);
  float* E32 = cv.take<float>((size_t)p * k);
  float* d32 = cv.take<float>(p);
  float* rinv32 = cv.take<float>(p);
  float* Gpart = cv.take<float>((size_t)nblk * kk);
  float* Fpart = cv.take<float>((size_t)nblk * kk);
  float* bpart = cv.take<float>((size_t)nblk * k);
  double* GFb = cv.take<double>(2 * kk + k);
  double* T = cv.take<double>(kk);
  float* T32 = cv.take<float>(kk);
  double* dsq_part = cv.take<double>(nprior);
  double* bg_part = cv.take<double>(nupd);
  double* an_part = cv.take<double>(nupd);
  double* sums = cv.take<double>(4);
  int* status = cv.take<int>(4);
  cudaStream_t s = ctx->stream;
  int rc;
  enkf_prior_mixed_kernel<<<nprior, kThreads, 0, s>>>(HX, yo, rvar, eps, p, k, Y32, E32, d32, rinv32, dsq_part);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  if ((rc = launch_cross<float>(ctx, Y32, Y32, rinv32, d32, p, k, nblk, per_block, Gpart, bpart)) != MG_OK ||
      (rc = launch_cross<float>(ctx, Y32, E32, rinv32, d32, p, k, nblk, per_block, Fpart, nullptr)) != MG_OK ||
      (rc = reduce_partials<float>(ctx, Gpart, nblk, kk, GFb)) != MG_OK ||
      (rc = reduce_partials<float>(ctx, Fpart, nblk, kk, GFb + kk)) != MG_OK ||
      (rc = reduce_partials<float>(ctx, bpart, nblk, k, GFb + 2 * kk)) != MG_OK)
    return rc;
  MG_TRY_CUDA(cudaMemsetAsync(status, 0, sizeof(int) * 4, s));
  MG_TRY_CUDA(mg::launch_enkf_chol(GFb, GFb + kk, GFb + 2 * kk, k, rho, T, T32, status, s));
  const size_t usmem = mg::upd_bytes(k);
  MG_TRY_CUDA(cudaFuncSetAttribute(enkf_update_mixed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)usmem));
  enkf_update_mixed_kernel<<<nupd, mg::kUpdThreads, usmem, s>>>(X, ld, n, k, T32, mean, bg_part, an_part);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  if (diag) {
    sum_partials_kernel<<<1, kThreads, 0, s>>>(dsq_part, nprior, sums + 0);
    sum_partials_kernel<<<1, kThreads, 0, s>>>(bg_part, nupd, sums + 1);
    sum_partials_kernel<<<1, kThreads, 0, s>>>(an_part, nupd, sums + 2);
    MG_COUNT_LAUNCH();
    MG_COUNT_LAUNCH();
    MG_COUNT_LAUNCH();
    MG_TRY_CUDA(cudaGetLastError());
  }
  return finish(ctx, n, k, rho, mean, mean_out, status, sums, diag);
}

}  // namespace

extern "C" int mg_enkf(mg_context* ctx, double* X, int64_t n, int32_t k, int64_t ld, const double* HX,
                       const double* yo, const double* rvar, const double* obs_pert, int64_t p, double inflation,
                       int32_t precision, double* mean_out, mg_enkf_diag* diag) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(X && n > 0 && k >= 2 && k <= 112 && ld >= n && p >= 1 && HX && yo && rvar && obs_pert &&
                   inflation > 0.0,
               "mg_enkf: bad arguments (k must be 2..112, p >= 1)");
  MG_CHECK_ARG(precision == MG_PREC_FP64 || precision == MG_PREC_MIXED, "mg_enkf: bad precision");
  if (precision == MG_PREC_FP64)
    return run_enkf_fp64(ctx, X, n, k, ld, HX, yo, rvar, obs_pert, p, inflation, mean_out, diag);
  return run_enkf_mixed(ctx, X, n, k, ld, HX, yo, rvar, obs_pert, p, inflation, mean_out, diag);
}
