// Observation operators (HX) and the obs-space prior (mean, anomalies,
// innovation).  Arithmetic that must be bit-identical to the reference uses
// explicitly rounded intrinsics so the compiler cannot contract a multiply
// and an add into one FMA.
#include <algorithm>
#include <cmath>

#include "mg_fp64.cuh"
#include "mg_internal.h"

namespace {

// IDW4 at integer grid coordinates (IdentityObsOperator.hpp:594-617, 2-D
// branch, and :643-676).  The four neighbours lie at distance 0, 1 or
// sqrt(2), or collapse onto each other at the grid's last column and row, so
// there are four weight sets, by (last column, last row); the host computes
// them with the reference's operations (IEEE square root and division).
struct Idw4Weights {
  double w[4][4];
  double wsum[4], rinv[4];  // rinv: 1 / wsum rounded
};

Idw4Weights idw4_weights() {
  Idw4Weights t;
  for (int c = 0; c < 4; ++c) {
    t.wsum[c] = 0.0;
    for (int q = 0; q < 4; ++q) {
      const double dx = (c & 1) ? 0.0 : (double)(q & 1), dy = (c & 2) ? 0.0 : (double)(q >> 1);
      const double dist = std::sqrt(dx * dx + dy * dy);
      t.w[c][q] = dist == 0.0 ? 1e12 : 1.0 / dist;
      t.wsum[c] += t.w[c][q];
    }
    t.rinv[c] = 1.0 / t.wsum[c];
  }
  return t;
}

// One thread per (obs, member).  Eight separately rounded FP64 operations for
// the weighted sum and a division: by Markstein's theorem (1990) one
// correction of ws * RN(1 / wsum) by its exact remainder is the correctly
// rounded quotient away from the ends of the exponent range, where the plain
// division is taken.  (The weights' square roots and divisions per value
// took 250 us for 20,000 obs x 64 members, now 34 us.)
__global__ void __launch_bounds__(256) hx_idw4_kernel(const double* __restrict__ X, int k, int64_t ld, int nx, int ny,
                                                      const int32_t* __restrict__ obs_xy,
                                                      const uint8_t* __restrict__ valid, int64_t p, Idw4Weights wt,
                                                      double* __restrict__ HX) {
  const int64_t total = p * k;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride) {
    const int64_t o = e / k;
    const int i = (int)(e - o * k);
    double v = 0.0;
    if (!valid || valid[o]) {
      const int i0 = max(0, min(nx - 1, obs_xy[2 * o])), j0 = max(0, min(ny - 1, obs_xy[2 * o + 1]));
      const int i1 = min(i0 + 1, nx - 1), j1 = min(j0 + 1, ny - 1);
      const int c = (i1 == i0) | (j1 == j0) << 1;
      const double* x = X + (int64_t)i * ld;
      const double x0 = __ldg(x + (int64_t)j0 * nx + i0), x1 = __ldg(x + (int64_t)j0 * nx + i1);
      const double x2 = __ldg(x + (int64_t)j1 * nx + i0), x3 = __ldg(x + (int64_t)j1 * nx + i1);
      double ws = __dadd_rn(0.0, __dmul_rn(wt.w[c][0], x0));
      ws = __dadd_rn(ws, __dmul_rn(wt.w[c][1], x1));
      ws = __dadd_rn(ws, __dmul_rn(wt.w[c][2], x2));
      ws = __dadd_rn(ws, __dmul_rn(wt.w[c][3], x3));
      const unsigned ex = ((unsigned)__double2hiint(ws) >> 20) & 0x7ff;
      v = (ex > 200 && ex < 2000) ? mg::div_refined(ws, wt.wsum[c], wt.rinv[c]) : __ddiv_rn(ws, wt.wsum[c]);
    }
    HX[e] = v;
  }
}

// Bilinear in (lon, lat), linear in level; the operation order matches the
// oracle's restatement exactly.
// TX: the members' storage type (FP64, or FP32 widened to FP64 on load).
//
// Each warp takes 32 obs.  Lane j first computes obs j's grid geometry
// (fractional indices, weights, plane offsets: about 30 FP64 operations,
// which GB300 runs at 1/64 of the FP32 rate) and leaves it in shared memory;
// then the warp walks the 32 obs with its lanes over the members, so the
// geometry is computed once per obs instead of once per (obs, member).
struct LatLonGeom {
  double ax, fx, ay, fy, az, fz;
  int64_t lo, hi;  // offsets of the two level planes from the member's start
  int64_t r0, r1;  // j0 nlon, (j0 + 1) nlon
  int32_t i0, i1;
  int32_t valid;
};

// The corners of the two planes, widened.
__device__ __forceinline__ void load8(double (&x)[8], const double* a, const double* b, const double* c,
                                      const double* d, int i0, int i1) {
  x[0] = a[i0]; x[1] = a[i1]; x[2] = b[i0]; x[3] = b[i1];
  x[4] = c[i0]; x[5] = c[i1]; x[6] = d[i0]; x[7] = d[i1];
}
// FP32 members: 21 FP64 instructions a value remain of 29 when the widening
// takes integer operations (64 members, 500k obs in random order: 2.95 -> 2.64 ms;
// the rest is 32-byte sectors from DRAM, four a value).
__device__ __forceinline__ void load8(double (&x)[8], const float* a, const float* b, const float* c, const float* d,
                                      int i0, int i1) {
  const float v[8] = {a[i0], a[i1], b[i0], b[i1], c[i0], c[i1], d[i0], d[i1]};
  bool special = false;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    special |= mg::wide_special(v[q]);
    x[q] = mg::wide(v[q]);
  }
  if (special) {
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = mg::wide_cvt(v[q]);
  }
}

template <typename TX>
__global__ void __launch_bounds__(256) hx_latlon_kernel(const TX* __restrict__ X, int k, int64_t ld, int nlon,
                                                        int nlat, int nlev, const double* __restrict__ olat,
                                                        const double* __restrict__ olon,
                                                        const double* __restrict__ olev,
                                                        const int32_t* __restrict__ ovar, int64_t p,
                                                        double* __restrict__ HX) {
  __shared__ LatLonGeom geo[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t plane = (int64_t)nlat * nlon;
  const int64_t nwarps = (int64_t)gridDim.x * 8;
  for (int64_t o0 = ((int64_t)blockIdx.x * 8 + w) * 32; o0 < p; o0 += nwarps * 32) {
    {
      const int64_t o = o0 + lane;
      LatLonGeom g{};
      // Reads stay inside member m: the variable must fit within the member
      // stride and the coordinates must be finite; otherwise the value is NaN.
      if (o < p && isfinite(olon[o]) && isfinite(olat[o]) && isfinite(olev[o]) && ovar[o] >= 0 &&
          ((int64_t)ovar[o] + 1) * nlev * plane <= ld) {
        // Fractional grid indices: lon_i = (i + 0.5) dlon, lat_j = -90 + (j + 0.5) dlat.
        const double dlon = 360.0 / (double)nlon, dlat = 180.0 / (double)nlat;
        const double gx = __dsub_rn(__ddiv_rn(olon[o], dlon), 0.5);
        const double fxl = floor(gx);
        const double fx = __dsub_rn(gx, fxl);
        long long i0 = (long long)fxl % nlon;
        if (i0 < 0) i0 += nlon;
        const long long i1 = (i0 + 1) % nlon;
        double gy = __dsub_rn(__ddiv_rn(__dadd_rn(olat[o], 90.0), dlat), 0.5);
        gy = fmax(0.0, fmin((double)(nlat - 1), gy));
        long long j0 = (long long)floor(gy);
        if (j0 > nlat - 2) j0 = nlat - 2;
        const double fy = __dsub_rn(gy, (double)j0);
        const double gz = fmax(0.0, fmin((double)(nlev - 1), olev[o]));
        long long l0 = (long long)floor(gz);
        if (l0 > nlev - 2) l0 = nlev - 2;
        if (l0 < 0) l0 = 0;
        const double fz = (nlev > 1) ? __dsub_rn(gz, (double)l0) : 0.0;
        const long long l1 = (nlev > 1) ? l0 + 1 : l0;
        const int64_t vb = (int64_t)ovar[o] * nlev * plane;
        g.ax = __dsub_rn(1.0, fx);
        g.fx = fx;
        g.ay = __dsub_rn(1.0, fy);
        g.fy = fy;
        g.az = __dsub_rn(1.0, fz);
        g.fz = fz;
        g.lo = vb + l0 * plane;
        g.hi = vb + l1 * plane;
        g.r0 = (int64_t)j0 * nlon;
        g.r1 = (int64_t)(j0 + 1) * nlon;
        g.i0 = (int32_t)i0;
        g.i1 = (int32_t)i1;
        g.valid = 1;
      }
      geo[w][lane] = g;
    }
    __syncwarp();
    const int nob = (p - o0 < 32) ? (int)(p - o0) : 32;
    for (int j = 0; j < nob; ++j) {
      const LatLonGeom& g = geo[w][j];
      const int64_t o = o0 + j;
      for (int m = lane; m < k; m += 32) {
        const int64_t e = o * k + m;
        if (!g.valid) {
          HX[e] = __longlong_as_double(0x7ff8000000000000LL);
          continue;
        }
        const TX* lo = X + (int64_t)m * ld + g.lo;
        const TX* hi = X + (int64_t)m * ld + g.hi;
        double x[8];
        load8(x, lo + g.r0, lo + g.r1, hi + g.r0, hi + g.r1, g.i0, g.i1);
        const double l00 = x[0], l01 = x[1], l10 = x[2], l11 = x[3];
        const double h00 = x[4], h01 = x[5], h10 = x[6], h11 = x[7];
        const double b0 = __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(l00, g.ax), __dmul_rn(l01, g.fx)), g.ay),
                                    __dmul_rn(__dadd_rn(__dmul_rn(l10, g.ax), __dmul_rn(l11, g.fx)), g.fy));
        const double b1 = __dadd_rn(__dmul_rn(__dadd_rn(__dmul_rn(h00, g.ax), __dmul_rn(h01, g.fx)), g.ay),
                                    __dmul_rn(__dadd_rn(__dmul_rn(h10, g.ax), __dmul_rn(h11, g.fx)), g.fy));
        HX[e] = __dadd_rn(__dmul_rn(b0, g.az), __dmul_rn(b1, g.fz));
      }
    }
    __syncwarp();
  }
}

// ym = (sum_i HX[o,i]) / k (rowwise().mean()), Y' = HX - ym, d = yo - ym,
// rinv = 1 / rvar.  A warp takes `rows` obs (32, fewer when that would leave
// SMs without a warp per scheduler): 1 / rvar for all of them at once,
// then the rows four at a time, their lane sums reduced together (each
// exchange halves the rows a lane carries, so four rows take six additions
// instead of twenty, in the same tree) and one division for the four means.
// FP64 warp instructions are what bounds this (64 cycles each): about six a
// row instead of fifty; 500,000 obs x 64 members 737 -> 289 us.
__global__ void __launch_bounds__(256) obs_prior_kernel(const double* __restrict__ HX, const double* __restrict__ yo,
                                                        const double* __restrict__ rvar, int64_t p, int k, int rows,
                                                        double* __restrict__ Y64, float* __restrict__ Y32,
                                                        double* __restrict__ d, double* __restrict__ rinv) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const double dk = (double)k, rk = 1.0 / dk;
  for (int64_t ob = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * rows; ob < p;
       ob += warps * rows) {
    const int nob = p - ob < rows ? (int)(p - ob) : rows;
    if (rinv && lane < nob) rinv[ob + lane] = 1.0 / rvar[ob + lane];
    const double yl = (d && lane < nob) ? yo[ob + lane] : 0.0;
    double dl = 0.0;  // d of obs ob + lane
    for (int q0 = 0; q0 < nob; q0 += 4) {
      double s[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        s[q] = 0.0;
        if (q0 + q < nob) {
          const double* h = HX + (ob + q0 + q) * k;
          for (int i = lane; i < k; i += 32) s[q] += h[i];
        }
      }
      // lane bit 4 keeps rows {0, 1} or {2, 3}, bit 3 one of the two
      const bool up = lane & 16, up2 = lane & 8;
      double a = up ? s[2] : s[0], b = up ? s[3] : s[1];
      a += __shfl_xor_sync(0xffffffffu, up ? s[0] : s[2], 16);
      b += __shfl_xor_sync(0xffffffffu, up ? s[1] : s[3], 16);
      double t = up2 ? b : a;
      t += __shfl_xor_sync(0xffffffffu, up2 ? a : b, 8);
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
      const unsigned ex = ((unsigned)__double2hiint(t) >> 20) & 0x7ff;
      const double ym = (ex > 200 && ex < 2000) ? mg::div_refined(t, dk, rk) : t / dk;  // row 2 (lane >> 4) + bit 3
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double m = __shfl_sync(0xffffffffu, ym, (q >> 1) * 16 + (q & 1) * 8);
        if (q0 + q >= nob) break;
        if (lane == q0 + q) dl = m;
        const int64_t r = (ob + q0 + q) * k;
        for (int i = lane; i < k; i += 32) {
          const double v = HX[r + i] - m;
          if (Y64) Y64[r + i] = v;
          if (Y32) Y32[r + i] = (float)v;
        }
      }
    }
    if (d && lane < nob) d[ob + lane] = yl - dl;
  }
}

inline unsigned grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 152 * 64) b = 152 * 64;
  if (b < 1) b = 1;
  return (unsigned)b;
}

}  // namespace

namespace mg {

cudaError_t launch_obs_prior(const double* HX, const double* yo, const double* rvar, int64_t p,
                             int k, double* Y64, float* Y32, double* d, double* rinv,
                             cudaStream_t s) {
  if (p <= 0) return cudaSuccess;
  const int rows = (int)std::max<int64_t>(4, std::min<int64_t>(32, p / (152 * 16) / 4 * 4));
  obs_prior_kernel<<<grid_for((p + rows - 1) / rows * 32, 256), 256, 0, s>>>(HX, yo, rvar, p, k, rows, Y64, Y32, d,
                                                                             rinv);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace mg

extern "C" {

int mg_hx_idw4(mg_context* ctx, const double* X, int32_t k, int64_t ld, int32_t nx, int32_t ny,
               const int32_t* obs_xy, const uint8_t* valid, int64_t p, double* HX) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(X && obs_xy && HX && k > 0 && nx > 0 && ny > 0 && p >= 0 && ld >= (int64_t)nx * ny,
               "mg_hx_idw4: bad arguments");
  if (p == 0) return MG_OK;
  hx_idw4_kernel<<<grid_for(p * k, 256), 256, 0, ctx->stream>>>(X, k, ld, nx, ny, obs_xy, valid, p,
                                                                idw4_weights(), HX);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  return MG_OK;
}

int mg_hx_latlon(mg_context* ctx, const double* X, int32_t k, int64_t ld, int32_t nlon,
                 int32_t nlat, int32_t nlev, const double* obs_lat, const double* obs_lon,
                 const double* obs_lev, const int32_t* obs_var, int64_t p, double* HX) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(X && obs_lat && obs_lon && obs_lev && obs_var && HX && k > 0 && nlon > 0 &&
                   nlat > 1 && nlev > 0 && p >= 0,
               "mg_hx_latlon: bad arguments");
  if (p == 0) return MG_OK;
  hx_latlon_kernel<double><<<grid_for((p + 31) / 32 * 32, 256), 256, 0, ctx->stream>>>(X, k, ld, nlon, nlat, nlev,
                                                                          obs_lat, obs_lon, obs_lev,
                                                                          obs_var, p, HX);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  return MG_OK;
}

int mg_hx_latlon_f32(mg_context* ctx, const float* X, int32_t k, int64_t ld, int32_t nlon,
                     int32_t nlat, int32_t nlev, const double* obs_lat, const double* obs_lon,
                     const double* obs_lev, const int32_t* obs_var, int64_t p, double* HX) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(X && obs_lat && obs_lon && obs_lev && obs_var && HX && k > 0 && nlon > 0 &&
                   nlat > 1 && nlev > 0 && p >= 0,
               "mg_hx_latlon_f32: bad arguments");
  if (p == 0) return MG_OK;
  hx_latlon_kernel<float><<<grid_for((p + 31) / 32 * 32, 256), 256, 0, ctx->stream>>>(X, k, ld, nlon, nlat, nlev,
                                                                         obs_lat, obs_lon, obs_lev,
                                                                         obs_var, p, HX);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  return MG_OK;
}

}  // extern "C"
