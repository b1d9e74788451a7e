// LETKF in the reference's order (LETKF.hpp:101, :152-243): grid points in
// row-major order, each analysed with the obs-space prior of the current,
// partly analysed members, written in place.
//
// The order leaves more freedom than one point after another.  Point g reads
// the members only at the cells that interpolate its local obs: analysed
// values at cells before g, background values at g and after.  With the
// background kept beside the analysis (both point-major), nothing is
// overwritten that a point still has to read, and g waits only for those of
// its cells that come before it.  CTAs take points from a counter in
// row-major order, wait on the cells' done flags and publish their own; a
// point's cells were taken earlier, by CTAs that are running or finished, so
// the waits end whatever the number of CTAs.  They are bounded as well: a wait
// gives up, with a status, when no point at all has been published for a
// time that covers the longest list (the last of the points in flight waits
// for all the others, however long that takes).
//
// A point on the critical chain is latency: the Gram's entries are spread
// over the CTA by output (packed lower triangle of A with Y'^T d as its last
// row, no idle lanes: a warp's FP64 instruction holds its scheduler 64
// cycles on GB300), the factorisation A = U D U^T needs one reciprocal per
// column and no inverse (mg_letkf_chol.cu explains the algebra), and for
// k <= 16 one warp runs it without CTA barriers.  Tutorial case (36 x 18
// points, k = 9, 28 obs, radius 10): 27.3 ms by one CTA walking all points,
// 0.83 ms for the whole cycle now.
#include <algorithm>

#include "mg_fp64.cuh"
#include "mg_internal.h"

namespace {

constexpr int kThreads = 128;
constexpr int kCh = 32;  // obs per chunk (four threads per obs in the row means)
// Time without a published point after which a wait gives up: 10 s, and 10 us
// an obs (a CTA takes 1.3 us at k = 64).
constexpr int64_t kWaitNs = 10ll * 1000 * 1000 * 1000, kWaitNsPerObs = 10000;

// Interpolation of one grid obs (IdentityObsOperator.hpp:594-676): four cells
// and inverse-distance weights; cell[0] < 0 marks an invalid obs (H = 0).
struct ObsStencil {
  int cell[4];
  double w[4];
  double wsum, rinv;
};

struct SeqParams {
  const double* Xb;  // background, point-major
  double* Xa;        // analysis, point-major
  int k, npt;
  const ObsStencil* st;
  const double* yo;
  const int64_t* loc_off;
  const int32_t* loc_idx;
  double rho;
  int* done;
  unsigned* next;
  int* status;
  int* gave_up;  // set where a wait did
  unsigned long long wait_ns;
};

__global__ void obs_stencil_kernel(const int32_t* __restrict__ obs_xy, const uint8_t* __restrict__ valid, int64_t p,
                                   int nx, int ny, ObsStencil* __restrict__ out) {
  const int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= p) return;
  ObsStencil s;
  const double xx = fmax(0.0, fmin((double)(nx - 1), (double)obs_xy[2 * o]));
  const double yy = fmax(0.0, fmin((double)(ny - 1), (double)obs_xy[2 * o + 1]));
  const int i0 = (int)floor(xx), j0 = (int)floor(yy);
  const int i1 = min(i0 + 1, nx - 1), j1 = min(j0 + 1, ny - 1);
  const int ii[4] = {i0, i1, i0, i1}, jj[4] = {j0, j0, j1, j1};
  s.wsum = 0.0;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const double dx = __dsub_rn(xx, (double)ii[t]), dy = __dsub_rn(yy, (double)jj[t]);
    const double dist = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
    s.w[t] = (dist == 0.0) ? 1e12 : __ddiv_rn(1.0, dist);
    s.wsum = __dadd_rn(s.wsum, s.w[t]);
    s.cell[t] = jj[t] * nx + ii[t];
  }
  s.rinv = __ddiv_rn(1.0, s.wsum);
  if (valid && !valid[o]) s.cell[0] = -1;
  out[o] = s;
}

// Member-major X -> point-major copy.
__global__ void __launch_bounds__(256) members_to_points_kernel(const double* __restrict__ X, int64_t n, int k,
                                                                int64_t ld, double* __restrict__ P) {
  __shared__ double tile[64][33];
  const int64_t s0 = (int64_t)blockIdx.x * 32;
  for (int e = threadIdx.x; e < 32 * k; e += 256) {
    const int i = e >> 5, j = e & 31;
    if (s0 + j < n) tile[i][j] = X[(int64_t)i * ld + s0 + j];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 32 * k; e += 256) {
    const int j = e / k, i = e - j * k;
    if (s0 + j < n) P[(s0 + j) * k + i] = tile[i][j];
  }
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Waits until the point is published; false when the time is up or another
// CTA has given up.  A CTA that publishes a point takes the next, so the points'
// counter moves with every published one.
__device__ bool wait_done(const int* flag, const unsigned* next, const int* gave_up, unsigned long long wait_ns) {
  if (ld_acquire(flag)) return true;
  unsigned long long t0 = now_ns();
  int seen = ld_acquire(reinterpret_cast<const int*>(next));
  for (;;) {
    for (int i = 0; i < 64; ++i)
      if (ld_acquire(flag)) return true;
    if (ld_acquire(gave_up) || now_ns() - t0 > wait_ns) return false;
    const int n = ld_acquire(reinterpret_cast<const int*>(next));
    if (n != seen) {
      seen = n;
      t0 = now_ns();
    }
  }
}

template <int KMAX>
__global__ void __launch_bounds__(kThreads) letkf_seq_kernel(SeqParams prm) {
  constexpr bool ONE = KMAX <= 16;  // factorisation and solves by the first warp alone
  constexpr int NOUT = (KMAX + 1) * (KMAX + 2) / 2 - 1;
  constexpr int OPT = (NOUT + kThreads - 1) / kThreads;  // outputs per thread
  constexpr int NV = KMAX <= 32 ? 1 : KMAX / 32;
  constexpr int LDY = KMAX + 1;
  __shared__ double P[NOUT + 1];  // rows i of the lower triangle, row k: b = Y'^T d
  __shared__ double Ys[kCh * LDY];
  __shared__ double raw[KMAX], dinv[KMAX], dval[KMAX], wa_s[KMAX], rs_s[KMAX], xb[KMAX];
  __shared__ const double* src[kCh * 4];
  __shared__ double s_xm;
  __shared__ unsigned s_item;
  __shared__ int s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = prm.k;
  const double rk = 1.0 / (double)k, dk = (double)k;
  const int nout = (k + 1) * (k + 2) / 2 - 1;
  // Fewer outputs than threads: the chunk's obs are split over `parts` threads per output.
  const int parts = nout <= kThreads / 4 ? 4 : (nout <= kThreads / 2 ? 2 : 1);
  const int width = kThreads / parts, part = tid / width;
  int oi[OPT], ol[OPT];
#pragma unroll
  for (int u = 0; u < OPT; ++u) {
    const int e = tid % width + u * kThreads;
    int i = 0;
    while ((i + 1) * (i + 2) / 2 <= e) ++i;
    oi[u] = e < nout ? i : -1;
    ol[u] = e - i * (i + 1) / 2;
  }
  const double cw = sqrt((double)(k - 1) * prm.rho);
  if (tid == 0) s_fail = 0;

  for (;;) {
    __syncthreads();
    if (tid == 0) s_item = atomicAdd(prm.next, 1u);
    __syncthreads();
    if (s_item >= (unsigned)prm.npt || s_fail) break;
    const int g = (int)s_item;
    const int64_t e0 = prm.loc_off[g], e1 = prm.loc_off[g + 1];
    if (tid < k) xb[tid] = prm.Xb[(int64_t)g * k + tid];
    double acc[OPT];
#pragma unroll
    for (int u = 0; u < OPT; ++u) acc[u] = 0.0;

    for (int64_t c0 = e0; c0 < e1; c0 += kCh) {
      const int cnt = (int)(e1 - c0 < (int64_t)kCh ? e1 - c0 : (int64_t)kCh);
      if (tid < cnt * 4) {
        const ObsStencil& s = prm.st[prm.loc_idx[c0 + (tid >> 2)]];
        const int c = s.cell[tid & 3];
        const double* q = nullptr;
        if (s.cell[0] >= 0) {
          if (c < g && !wait_done(prm.done + c, prm.next, prm.gave_up, prm.wait_ns)) s_fail = 1;
          q = (c < g ? prm.Xa : prm.Xb) + (int64_t)c * k;
        }
        src[tid] = q;
      }
      __syncthreads();
      // H of the current members (LETKF.hpp:197-206)
      for (int e = tid; e < cnt * k; e += kThreads) {
        const int r = e / k, i = e - r * k;
        const ObsStencil& s = prm.st[prm.loc_idx[c0 + r]];
        double v = 0.0;
        if (src[4 * r]) {
          double ws = 0.0;
#pragma unroll
          for (int q = 0; q < 4; ++q) ws = __dadd_rn(ws, __dmul_rn(s.w[q], __ldcg(src[4 * r + q] + i)));
          v = mg::div_refined(ws, s.wsum, s.rinv);
        }
        Ys[r * LDY + i] = v;
      }
      __syncthreads();
      {  // row mean, anomalies, innovation (:209-211): four threads per obs
        const int r = tid >> 2, q = tid & 3;
        double s = 0.0;
        if (r < cnt)
          for (int j = q; j < k; j += 4) s += Ys[r * LDY + j];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        const double ym = mg::div_refined(s, dk, rk);
        if (r < cnt) {
          for (int j = q; j < k; j += 4) Ys[r * LDY + j] -= ym;
          if (q == 0) Ys[r * LDY + k] = prm.yo[prm.loc_idx[c0 + r]] - ym;
        }
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < OPT; ++u) {
        if (oi[u] < 0) continue;
        const double *yi = Ys + oi[u], *yl = Ys + ol[u];
        for (int r = part; r < cnt; r += parts) acc[u] = __fma_rn(yi[r * LDY], yl[r * LDY], acc[u]);
      }
      __syncthreads();
    }
    __syncthreads();  // xb, where there was no chunk
    if (s_fail) break;
    if (warp == 3) {  // own mean (:154-157)
      double s = 0.0;
      for (int i = lane; i < k; i += 32) s += xb[i];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      if (lane == 0) s_xm = mg::div_refined(s, dk, rk);
    }
    if (e1 > e0) {
      if (parts > 1) {  // sum the parts through Ys (free now): parts * width = kThreads values
        Ys[tid] = acc[0];
        __syncthreads();
        if (part == 0)
          for (int q = 1; q < parts; ++q) acc[0] += Ys[tid + q * width];
      }
      if (part == 0) {
#pragma unroll
        for (int u = 0; u < OPT; ++u)
          if (oi[u] >= 0) P[tid + u * kThreads] = acc[u] + (oi[u] == ol[u] ? (double)(k - 1) : 0.0);
      }
      __syncthreads();
      // ---- A = U D U^T from the last column up; b <- U^-1 b as row k ----
      auto sync = [] {
        if (ONE) __syncwarp();
        else __syncthreads();
      };
      if (!ONE || warp == 0) {
        constexpr int NT = ONE ? 32 : kThreads;
        double* const b = P + k * (k + 1) / 2;
        bool ok = true;
        for (int j = k - 1; j >= 0; --j) {
          double* const rw = P + j * (j + 1) / 2;
          double d = rw[j];
          if (!mg::pivot_ok(d)) {
            ok = false;
            d = 1.0;
          }
          const double r = mg::recip_fp64(d);
          const double uk = b[j] * r;
          for (int l = tid; l < j; l += NT) {
            const double a = rw[l];
            raw[l] = a;
            rw[l] = a * r;
          }
          if (tid == 0) {
            dinv[j] = r;
            dval[j] = d;
          }
          sync();
          const int ne = j * (j + 1) / 2;  // rows below j, then row k's first j entries
          for (int e = tid; e < ne + j; e += NT) {
            if (e < ne) {
              int i = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
              if ((i + 1) * (i + 2) / 2 <= e) ++i;
              if (i * (i + 1) / 2 > e) --i;
              P[e] = __fma_rn(-rw[i], raw[e - i * (i + 1) / 2], P[e]);
            } else {
              b[e - ne] = __fma_rn(-uk, raw[e - ne], b[e - ne]);
            }
          }
          sync();
        }
        if (!ok && tid == 0) atomicExch(prm.status, 1);
        // ---- wa = U^-T D^-1 z, row sums of M = U^-T D^-1/2 1 ----
        if (ONE || warp < 2) {
          const bool dw = ONE || warp == 0, dr = ONE || warp == 1;
          double x[NV], y[NV];
#pragma unroll
          for (int m = 0; m < NV; ++m) {
            const int i = lane + 32 * m;
            x[m] = (dw && i < k) ? b[i] * dinv[i] : 0.0;
            y[m] = (dr && i < k) ? rsqrt(dval[i]) : 0.0;
          }
#pragma unroll
          for (int m = 0; m < NV; ++m) {
            for (int ll = 0; ll < 32; ++ll) {
              const int l = 32 * m + ll;
              if (l >= k - 1) break;
              const double xl = __shfl_sync(0xffffffffu, x[m], ll), yl = __shfl_sync(0xffffffffu, y[m], ll);
#pragma unroll
              for (int q = m; q < NV; ++q) {
                const int i = lane + 32 * q;
                if (i > l && i < k) {
                  const double s = P[i * (i + 1) / 2 + l];
                  if (dw) x[q] = __fma_rn(-s, xl, x[q]);
                  if (dr) y[q] = __fma_rn(-s, yl, y[q]);
                }
              }
            }
          }
#pragma unroll
          for (int m = 0; m < NV; ++m) {
            const int i = lane + 32 * m;
            if (i < k) {
              if (dw) wa_s[i] = prm.rho * x[m];
              if (dr) rs_s[i] = cw * y[m];
            }
          }
        }
      }
    }
    __syncthreads();
    if (tid < k) {
      const double xm = s_xm, xp = xb[tid] - xm;
      // :227-242, and without local obs :167-190
      const double xa = e1 > e0 ? (xm + xp * wa_s[tid]) + xp * rs_s[tid] : xm + xp * sqrt(prm.rho);
      __stcg(prm.Xa + (int64_t)g * k + tid, xa);
    }
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(prm.done + g), "r"(1) : "memory");
    }
  }
  if (s_fail && tid == 0) atomicExch(prm.gave_up, 1);
}

template <int KMAX>
cudaError_t launch_seq(const SeqParams& prm, int num_sms, cudaStream_t s) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, letkf_seq_kernel<KMAX>, kThreads, 0);
  if (e != cudaSuccess) return e;
  const int grid = std::min(prm.npt, std::max(1, std::min(per_sm, 4)) * num_sms);
  letkf_seq_kernel<KMAX><<<grid, kThreads, 0, s>>>(prm);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

int compat_grid(mg_context* ctx, double* X, int32_t k, int64_t ld, int32_t nx, int32_t ny, const int32_t* obs_xy,
                const uint8_t* valid, const double* yo, int64_t p, double radius, double rho, double* mean_out,
                int64_t wait_ns) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(X && k >= 2 && k <= 64 && nx > 0 && ny > 0 && ld >= (int64_t)nx * ny && p >= 0 &&
                   (p == 0 || (obs_xy && yo)) && rho > 0.0,
               "mg_letkf_compat_grid: bad arguments (k must be 2..64)");
  const int64_t npt = (int64_t)nx * ny;
  MG_CHECK_ARG(npt < ((int64_t)1 << 31), "mg_letkf_compat_grid: grid too large");
  // One workspace holds the search's scratch (at its start, where
  // mg_select_grid carves it) and what this call keeps; the lists take what
  // is left of it, and the search runs again only when they do not fit.
  const size_t sel = mg::select_grid_bytes(npt);
  int64_t total = 0, cap = 0;
  mg::Carver cv;
  int64_t* off = nullptr;
  int32_t* idx = nullptr;
  double *Xb = nullptr, *Xa = nullptr;
  ObsStencil* st = nullptr;
  int* done = nullptr;
  int* flags = nullptr;
  for (int attempt = 0;; ++attempt) {
    cv = mg::Carver{};
    cv.reserve<char>(sel);
    cv.reserve<double>((size_t)npt * k);
    cv.reserve<double>((size_t)npt * k);
    cv.reserve<ObsStencil>((size_t)p + 1);
    cv.reserve<int>((size_t)npt);
    cv.reserve<int>(4);
    cv.reserve<int64_t>((size_t)npt + 1);
    const size_t fixed = cv.off + 256;
    if (attempt == 0) cap = ctx->ws_bytes > fixed ? (int64_t)((ctx->ws_bytes - fixed) / sizeof(int32_t)) : 1;
    else cap = total;
    cv.reserve<int32_t>((size_t)cap);
    void* ws = mg::workspace(ctx, cv.off);
    if (!ws) return MG_ERR_NOMEM;
    cv = mg::Carver{static_cast<char*>(ws), 0};
    cv.take<char>(sel);
    Xb = cv.take<double>((size_t)npt * k);
    Xa = cv.take<double>((size_t)npt * k);
    st = cv.take<ObsStencil>((size_t)p + 1);
    done = cv.take<int>((size_t)npt);
    flags = cv.take<int>(4);  // next, status, gave up
    off = cv.take<int64_t>((size_t)npt + 1);
    idx = cv.take<int32_t>((size_t)cap);
    const int rc = mg_select_grid(ctx, nx, ny, obs_xy, p, radius, off, idx, cap, &total);
    if (rc == MG_OK) break;
    if (rc != MG_ERR_CAPACITY || attempt > 0) return rc;
  }
  cudaStream_t s = ctx->stream;
  MG_TRY_CUDA(cudaMemsetAsync(done, 0, sizeof(int) * npt, s));
  MG_TRY_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * 4, s));
  if (p > 0) {
    obs_stencil_kernel<<<(unsigned)((p + 127) / 128), 128, 0, s>>>(obs_xy, valid, p, nx, ny, st);
    MG_COUNT_LAUNCH();
  }
  members_to_points_kernel<<<(unsigned)((npt + 31) / 32), 256, 0, s>>>(X, npt, k, ld, Xb);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  const SeqParams prm{Xb, Xa, k, (int)npt, st, yo, off, idx, rho, done, reinterpret_cast<unsigned*>(flags), flags + 1,
                      flags + 2, (unsigned long long)wait_ns};
  if (k <= 16) MG_TRY_CUDA(launch_seq<16>(prm, ctx->num_sms, s));
  else if (k <= 32) MG_TRY_CUDA(launch_seq<32>(prm, ctx->num_sms, s));
  else MG_TRY_CUDA(launch_seq<64>(prm, ctx->num_sms, s));
  // A run that gave up has points without an analysis: the members and the mean stay as they are.
  MG_TRY_CUDA(mg::launch_point_major_to_members(Xa, npt, k, X, ld, s, prm.gave_up));
  if (mean_out)
    MG_TRY_CUDA(mg::launch_mean_pert_members(X, npt, k, ld, mean_out, nullptr, nullptr, 0, s, prm.gave_up));
  int* hs = static_cast<int*>(mg::host_stage(ctx, 2 * sizeof(int)));  // pinned
  if (!hs) return MG_ERR_NOMEM;
  MG_TRY_CUDA(cudaMemcpyAsync(hs, flags + 1, 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
  MG_TRY_CUDA(cudaStreamSynchronize(s));
  if (hs[1]) return mg::fail(ctx, MG_ERR_TIMEOUT, "mg_letkf_compat_grid: a bounded wait for an earlier point gave up");
  if (hs[0] != 0)
    return mg::fail(ctx, MG_ERR_NUMERIC, "mg_letkf_compat_grid: a local k x k system was not positive definite");
  return MG_OK;
}

}  // namespace

extern "C" {

int mg_letkf_compat_grid(mg_context* ctx, double* X, int32_t k, int64_t ld, int32_t nx, int32_t ny,
                         const int32_t* obs_xy, const uint8_t* valid, const double* yo, int64_t p, double radius,
                         double rho, double* mean_out) {
  return compat_grid(ctx, X, k, ld, nx, ny, obs_xy, valid, yo, p, radius, rho, mean_out,
                     kWaitNs + kWaitNsPerObs * p);
}

int mg_letkf_compat_grid_wait_selftest(mg_context* ctx, double* X, int32_t k, int64_t ld, int32_t nx, int32_t ny,
                                       const int32_t* obs_xy, const uint8_t* valid, const double* yo, int64_t p,
                                       double radius, double rho, double* mean_out, int64_t wait_ns) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(wait_ns >= 0, "mg_letkf_compat_grid_wait_selftest: wait_ns must not be negative");
  return compat_grid(ctx, X, k, ld, nx, ny, obs_xy, valid, yo, p, radius, rho, mean_out, wait_ns);
}

}  // extern "C"
