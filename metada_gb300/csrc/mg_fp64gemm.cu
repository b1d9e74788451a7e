// FP64 contractions of the global analyses (ETKF.hpp:128-179, EnKF.hpp:168-225)
// on the tensor cores (mg_ozaki.cuh): the obs-space products
//   G = Y'^T R^-1 Y',  b = Y'^T R^-1 d  and, for the EnKF,  F = Y'^T R^-1 eps
// straight from H(X), and the state update Xa = xm 1^T + X' T (n x k).
#include <algorithm>

#include "mg_fp64.cuh"
#include "mg_internal.h"
#include "mg_ozaki.cuh"

namespace {

namespace oz = mg::oz;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kObs = 64;  // unit of a CTA's obs range

// -------------------------------------------------------------- obs space --
// Obs chunks of a contiguous range per CTA.  The obs-space prior is formed on
// the way (row means, Y' = HX - ym, d = yo - ym: no p x k buffer and no pass
// of its own).  Rows are whitened by 1/sigma (one FP64 multiplication per
// entry), each column gets its own scale, and a 16 x 8 tile's integer sum
// over the chunk is added to the FP64 accumulator its lanes keep for the
// CTA's whole range (two FP64 operations per entry and chunk, against 64
// multiply-adds).  G: the tiles that touch the lower triangle, with the
// innovation as one more column; F: all tiles.
//
// What the scaled integers cannot hold (non-finite values, magnitudes past
// 2^478, a negative sigma^2) is summed by the plain FP64 loop, chunk by chunk.
// 500,000 obs x 64 members: prior 0.74 ms and two products 4.52 + 4.39 ms on
// the FP64 units -> 1.35 ms; 1024 obs x 32 members 139 -> 13 us.
template <int KP, bool WITH_F>
struct ObsCfg {
  static constexpr int NT = WITH_F ? 512 : 256;
  // Obs per chunk: 64 rows of both operands fit one CTA (16 warps) per SM up
  // to k = 64 (two CTAs with 32 rows flush twice as often: 1.40 against
  // 1.35 ms at 500,000 obs x 64 members).
  static constexpr int OBS = (WITH_F && KP > 64) ? 32 : 64;
  static constexpr int LDO = OBS + 8;  // digit row stride in halves: 16-byte rows, conflict-free ldmatrix
  static constexpr int WARPS = NT / 32;
  static constexpr int MT = KP / 16;
  static constexpr int GT = MT * (MT + 1) + MT, FT = WITH_F ? MT * (KP / 8) : 0;
  static constexpr int TPW = (GT + FT + WARPS - 1) / WARPS;
  static constexpr int VROWS = 8 + (WITH_F ? KP : 0);    // digit rows beside Y's: the innovation, eps
  static constexpr size_t BYTES = sizeof(__half) * oz::kSlices * (KP + VROWS) * LDO + sizeof(double) * OBS * 3 +
                                  sizeof(int) * (2 * KP + 4);
};

// Also, where mean_blocks > 0, the ensemble mean of a small state, by the
// last mean_blocks CTAs (one launch less).
template <int KP, bool WITH_F>
__global__ void __launch_bounds__(ObsCfg<KP, WITH_F>::NT)
    obs_products_kernel(const double* __restrict__ HX, const double* __restrict__ eps, const double* __restrict__ yo,
                        const double* __restrict__ rvar, int64_t p, int k, int64_t per_block,
                        double* __restrict__ part, double* __restrict__ dsq_part, int mean_blocks,
                        const double* __restrict__ X, int64_t n, int64_t ld, double rk, double* __restrict__ mean) {
  using C = ObsCfg<KP, WITH_F>;
  constexpr int NT = C::NT;
  constexpr int SU = KP * C::LDO, SV = C::VROWS * C::LDO;  // slice strides
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = gridDim.x - mean_blocks;
  if ((int)blockIdx.x >= nblk) {  // Ensemble::RecomputeMean (member order)
    for (int64_t s = (int64_t)((int)blockIdx.x - nblk) * NT + tid; s < n; s += (int64_t)mean_blocks * NT) {
      double m = 0.0;
#pragma unroll 8
      for (int i = 0; i < k; ++i) m = __dadd_rn(m, X[(int64_t)i * ld + s]);
      mean[s] = __dmul_rn(m, rk);
    }
    return;
  }
  __half* dU = reinterpret_cast<__half*>(smem_raw);
  __half* dV = dU + oz::kSlices * SU;
  double* sw = reinterpret_cast<double*>(dV + oz::kSlices * SV);  // 1/sigma
  double* sd = sw + C::OBS;                                         // d/sigma
  double* ym = sd + C::OBS;
  int* exU = reinterpret_cast<int*>(ym + C::OBS);
  int* exE = exU + KP;
  int* exd = exE + KP;
  int* odd = exd + 1;
  const int64_t o0 = (int64_t)blockIdx.x * per_block, o1 = min(p, o0 + per_block);
  const double dk = (double)k;
  // The warp's tiles: (row tile, column tile, kind).
  enum { NONE = -1, GRAM = 0, INNOV = 1, CROSS = 2 };
  int tm[C::TPW], tn[C::TPW], tk[C::TPW];
#pragma unroll
  for (int u = 0; u < C::TPW; ++u) {
    int e = warp + u * C::WARPS;
    tm[u] = tn[u] = 0;
    tk[u] = NONE;
    if (e < C::GT) {
      int m = 0;
      while (e >= 2 * (m + 1) + 1) e -= 2 * (m + 1) + 1, ++m;
      tm[u] = m;
      tn[u] = e;
      tk[u] = e < 2 * (m + 1) ? GRAM : INNOV;
    } else if (e < C::GT + C::FT) {
      e -= C::GT;
      tm[u] = e / (KP / 8);
      tn[u] = e % (KP / 8);
      tk[u] = CROSS;
    }
  }
  double c64[C::TPW][4];
#pragma unroll
  for (int u = 0; u < C::TPW; ++u)
#pragma unroll
    for (int e = 0; e < 4; ++e) c64[u][e] = 0.0;
  double dsq = 0.0;

  // Digits of a chunk's whitened columns: items (column, eight obs).
  auto digits = [&](const double* A, bool anomalies, __half* dst, int stride, int* ex, int64_t c0) {
    constexpr int ITEMS = KP * (C::OBS / 8), PER = (ITEMS + NT - 1) / NT;
    double v[PER][8];
#pragma unroll
    for (int x = 0; x < PER; ++x) {
      const int it = tid + x * NT, i = it % KP, og = it / KP;
      if (it >= ITEMS) continue;
      int ef = 1;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int r = og * 8 + q;
        const double a = (i < k && c0 + r < o1) ? A[(c0 + r) * k + i] : 0.0;
        v[x][q] = (anomalies ? (i < k ? a - ym[r] : 0.0) : a) * sw[r];
        ef = max(ef, oz::ef_of(v[x][q]));
      }
      atomicMax(&ex[i], ef);
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < PER; ++x) {
      const int it = tid + x * NT, i = it % KP, og = it / KP;
      if (it >= ITEMS) continue;
      const int ef = ex[i];
      if (ef > oz::kMaxEf) *odd = 1;
      oz::store_digits8(v[x], ef, dst + i * C::LDO + og * 8, stride);
    }
  };

  for (int64_t c0 = o0; c0 < o1; c0 += C::OBS) {
    for (int i = tid; i < 2 * KP + 2; i += NT) exU[i] = i == 2 * KP + 1 ? 0 : 1;
    if (tid < C::OBS) sw[tid] = c0 + tid < o1 ? rsqrt(rvar[c0 + tid]) : 0.0;  // not finite where sigma^2 <= 0
    // row means: four rows of a warp reduced together (as obs_prior_kernel)
    for (int r0 = warp * 4; r0 < C::OBS; r0 += C::WARPS * 4) {
      double s[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        s[q] = 0.0;
        if (c0 + r0 + q < o1)
          for (int i = lane; i < k; i += 32) s[q] += HX[(c0 + r0 + q) * k + i];
      }
      const bool up = lane & 16, up2 = lane & 8;
      double a = up ? s[2] : s[0], b = up ? s[3] : s[1];
      a += __shfl_xor_sync(0xffffffffu, up ? s[0] : s[2], 16);
      b += __shfl_xor_sync(0xffffffffu, up ? s[1] : s[3], 16);
      double t = up2 ? b : a;
      t += __shfl_xor_sync(0xffffffffu, up2 ? a : b, 8);
#pragma unroll
      for (int off = 4; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
      const int ex = oz::ef_of(t);
      if ((lane & 7) == 0) ym[r0 + (lane >> 3)] = (ex > 200 && ex < 2000) ? mg::div_refined(t, dk, rk) : t / dk;
    }
    __syncthreads();
    if (tid < C::OBS) {
      if (oz::ef_of(sw[tid]) > oz::kMaxEf) *odd = 1;
      const double di = c0 + tid < o1 ? yo[c0 + tid] - ym[tid] : 0.0;
      if (dsq_part) dsq = __fma_rn(di, di, dsq);
      const double d = di * sw[tid];
      sd[tid] = d;
      atomicMax(exd, oz::ef_of(d));
    }
    digits(HX, true, dU, SU, exU, c0);
    if (tid < C::OBS) {  // eight columns, the innovation in the first
      const int i = tid & 7, og = tid >> 3;
      double v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = i == 0 ? sd[og * 8 + q] : 0.0;
      const int ef = *exd;
      if (ef > oz::kMaxEf) *odd = 1;
      oz::store_digits8(v, ef, dV + i * C::LDO + og * 8, SV);
    }
    if (WITH_F) digits(eps, false, dV + 8 * C::LDO, SV, exE, c0);
    __syncthreads();
    const bool plain = *odd != 0;
#pragma unroll
    for (int u = 0; u < C::TPW; ++u) {
      if (tk[u] == NONE) continue;
      const bool gram = tk[u] == GRAM, innov = tk[u] == INNOV;
      float acc[oz::kSlices][4];
      if (!plain)
        oz::tile<C::OBS / 16>(acc, dU + tm[u] * 16 * C::LDO, C::LDO, SU,
                            gram ? dU + tn[u] * 8 * C::LDO : (innov ? dV : dV + (8 + tn[u] * 8) * C::LDO), C::LDO,
                            gram ? SU : SV);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = tm[u] * 16 + (lane >> 2) + 8 * (e >> 1), jl = 2 * (lane & 3) + (e & 1), j = tn[u] * 8 + jl;
        if (!plain) {
          const int ev = innov ? *exd : (gram ? exU : exE)[j];
          c64[u][e] = __fma_rn((double)oz::combine(acc, e), oz::unit(exU[i], ev), c64[u][e]);
        } else if (i < k && (innov ? jl == 0 : j < k)) {
          double t = 0.0;
          for (int r = 0; r < C::OBS && c0 + r < o1; ++r) {
            const double* h = HX + (c0 + r) * k;
            const double v = innov ? yo[c0 + r] - ym[r] : (gram ? h[j] - ym[r] : eps[(c0 + r) * k + j]);
            t += ((h[i] - ym[r]) * (1.0 / rvar[c0 + r])) * v;
          }
          c64[u][e] += t;
        }
      }
    }
    __syncthreads();
  }
  const int64_t kk = (int64_t)k * k;
  double* out = part + (size_t)blockIdx.x * (kk + k + (WITH_F ? kk : 0));
#pragma unroll
  for (int u = 0; u < C::TPW; ++u) {
    if (tk[u] == NONE) continue;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = tm[u] * 16 + (lane >> 2) + 8 * (e >> 1), jl = 2 * (lane & 3) + (e & 1), j = tn[u] * 8 + jl;
      if (i >= k) continue;
      if (tk[u] == INNOV) {
        if (jl == 0) out[kk + i] = c64[u][e];
      } else if (tk[u] == CROSS) {
        if (j < k) out[kk + k + i * k + j] = c64[u][e];
      } else if (j <= i) {
        out[i * k + j] = c64[u][e];
        out[j * k + i] = c64[u][e];
      }
    }
  }
  if (dsq_part) {  // sum of squared innovations (threads 0 .. 63 hold it)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) dsq += __shfl_xor_sync(0xffffffffu, dsq, off);
    if (lane == 0 && warp < 2) sw[warp] = dsq;  // warp 1 holds zero where OBS is 32
    __syncthreads();
    if (tid == 0) dsq_part[blockIdx.x] = sw[0] + sw[1];
  }
}

template <int KP, bool WITH_F>
cudaError_t run_obs(const mg::ObsProducts& a, int mean_blocks, cudaStream_t s) {
  using C = ObsCfg<KP, WITH_F>;
  static_assert(C::BYTES <= 227 * 1024 && kObs % C::OBS == 0, "a CTA's shared memory");
  const cudaError_t e = cudaFuncSetAttribute(obs_products_kernel<KP, WITH_F>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::BYTES);
  if (e != cudaSuccess) return e;
  const int64_t chunks = (a.p + kObs - 1) / kObs, per_block = (chunks + a.nblk - 1) / a.nblk * kObs;
  obs_products_kernel<KP, WITH_F><<<a.nblk + mean_blocks, C::NT, C::BYTES, s>>>(
      a.HX, a.eps, a.yo, a.rvar, a.p, a.k, per_block, a.part, a.dsq_part, mean_blocks, a.X, a.n, a.ld,
      1.0 / (double)a.k, a.mean);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

template <bool WITH_F>
cudaError_t obs_by_k(const mg::ObsProducts& a, int mean_blocks, cudaStream_t s) {
  if (a.k <= 16) return run_obs<16, WITH_F>(a, mean_blocks, s);
  if (a.k <= 32) return run_obs<32, WITH_F>(a, mean_blocks, s);
  if (a.k <= 64) return run_obs<64, WITH_F>(a, mean_blocks, s);
  return run_obs<112, WITH_F>(a, mean_blocks, s);
}

// out[e] = sum of element e over the nblk partials: eight threads per element,
// each summing every eighth partial in order, then in thread order.  out may
// be the first partial: an element is read only by the CTA that writes it.
__global__ void __launch_bounds__(kThreads) reduce_parts_kernel(const double* part, int nblk, int64_t len,
                                                                double* out) {
  const int64_t e = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
  const int q = threadIdx.x >> 5;
  __shared__ double red[8][33];
  double t = 0.0;
  if (e < len)
    for (int b = q; b < nblk; b += 8) t += part[(size_t)b * len + e];
  red[q][threadIdx.x & 31] = t;
  __syncthreads();
  if (q == 0 && e < len) {
#pragma unroll
    for (int x = 1; x < 8; ++x) t += red[x][threadIdx.x];
    out[e] = t;
  }
}

// ------------------------------------------------------------------ update --
// Tiles of NS states.  A thread reads eight members of one state (lanes over
// consecutive states), subtracts the mean and writes the digits; T's digits
// (rows: output member, contracted over j) are made once per CTA.  Per value
// the FP64 pipe runs three operations (subtraction, integer conversion, one
// multiply-add that scales and adds the mean) instead of k; 2.59M states x 64
// members: 17.3 ms, and 0.66 ms for the X' it needed in memory -> 2.08 ms.
template <int KP>
struct UpdCfg {
  static constexpr int NS = KP <= 16 ? 128 : (KP <= 32 ? 64 : (KP <= 96 ? 32 : 16));
  static constexpr int LD = KP + 8;
  static constexpr int ITEMS = NS * (KP / 8), PER = (ITEMS + kThreads - 1) / kThreads;
  static constexpr int MT = KP / 16, TILES = MT * (NS / 8);
  static constexpr int OUT = (NS * KP + kThreads - 1) / kThreads;
  static constexpr size_t BYTES = sizeof(__half) * oz::kSlices * (KP + NS) * LD + sizeof(double) * NS +
                                  sizeof(int) * (KP + NS + 4);
};

// Any of the eight values not zero, by integer operations.
__device__ __forceinline__ bool any_nonzero(const double (&v)[8]) {
  long long b = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) b |= __double_as_longlong(v[q]);
  return (b << 1) != 0;
}

template <int KP>
__global__ void __launch_bounds__(kThreads) update_kernel(double* X, int64_t ld, int64_t n, int k,
                                                          const double* __restrict__ mean,
                                                          const double* __restrict__ T) {
  using C = UpdCfg<KP>;
  constexpr int NS = C::NS, LD = C::LD;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __half* dT = reinterpret_cast<__half*>(smem_raw);  // [slice][i][j]
  __half* dX = dT + oz::kSlices * KP * LD;           // [slice][s][j]
  double* sm = reinterpret_cast<double*>(dX + oz::kSlices * NS * LD);
  int* exT = reinterpret_cast<int*>(sm + NS);
  int* exX = exT + KP;
  int* odd = exX + NS;  // [0]: this tile, [1]: T, [2]: T's smallest row exponent
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < KP; i += kThreads) exT[i] = 1;
  if (tid < 3) odd[tid] = tid == 2 ? 0x7ff : 0;
  __syncthreads();
  for (int it = tid; it < KP * (KP / 8); it += kThreads) {
    const int i = it % KP, jg = it / KP;
    int ef = 1;
    for (int q = 0; q < 8; ++q)
      if (i < k && jg * 8 + q < k) ef = max(ef, oz::ef_of(T[(jg * 8 + q) * k + i]));
    atomicMax(&exT[i], ef);
  }
  __syncthreads();
  for (int it = tid; it < KP * (KP / 8); it += kThreads) {
    const int i = it % KP, jg = it / KP;
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = (i < k && jg * 8 + q < k) ? T[(jg * 8 + q) * k + i] : 0.0;
    if (exT[i] > oz::kMaxEf) odd[1] = 1;
    if (i < k) atomicMin(&odd[2], exT[i]);
    oz::store_digits8(v, exT[i], dT + i * LD + jg * 8, KP * LD);
  }
  __syncthreads();
  const int tiny = oz::kUnitEf - odd[2];  // exponents up to it: products below unit()'s (states of 1e-260 and less)
  const bool pair_ok = ((ld & 1) | ((reinterpret_cast<uintptr_t>(X) >> 3) & 1)) == 0;
  const int64_t ntiles = (n + NS - 1) / NS;
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t s0 = tile * NS;
    double v[C::PER][8];
#pragma unroll
    for (int x = 0; x < C::PER; ++x) {
      const int it = tid + x * kThreads;
      const int64_t s = s0 + it % NS;
      const int jg = it / NS;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        v[x][q] = (it < C::ITEMS && s < n && jg * 8 + q < k) ? X[(int64_t)(jg * 8 + q) * ld + s] : 0.0;
    }
    __syncthreads();  // the previous tile's readers are done
    if (tid < NS) {
      exX[tid] = 1;
      sm[tid] = s0 + tid < n ? mean[s0 + tid] : 0.0;
    }
    if (tid == 0) odd[0] = odd[1];
    __syncthreads();
#pragma unroll
    for (int x = 0; x < C::PER; ++x) {
      const int it = tid + x * kThreads;
      if (it >= C::ITEMS) continue;
      const int sl = it % NS, jg = it / NS;
      const double m = sm[sl];
      int ef = 1;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (jg * 8 + q < k) {
          v[x][q] -= m;
          ef = max(ef, oz::ef_of(v[x][q]));
        }
      }
      atomicMax(&exX[sl], ef);
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < C::PER; ++x) {
      const int it = tid + x * kThreads;
      if (it >= C::ITEMS) continue;
      const int sl = it % NS, jg = it / NS;
      const int ef = exX[sl];
      if ((unsigned)(ef - tiny - 1) >= (unsigned)(oz::kMaxEf - tiny) && (ef > tiny || any_nonzero(v[x]))) odd[0] = 1;
      oz::store_digits8(v[x], ef, dX + sl * LD + jg * 8, NS * LD);
    }
    __syncthreads();
    if (odd[0]) {  // magnitudes that the integers or their unit cannot hold: the plain FP64 sum
      double out[C::OUT];
#pragma unroll
      for (int u = 0; u < C::OUT; ++u) {
        const int e = tid + u * kThreads, i = e / NS, sl = e % NS;
        const int64_t s = s0 + sl;
        double acc = 0.0;
        if (i < k && s < n)
          for (int j = 0; j < k; ++j) acc += (X[(int64_t)j * ld + s] - sm[sl]) * T[j * k + i];
        out[u] = sm[sl] + acc;
      }
      __syncthreads();  // every read of the tile done
#pragma unroll
      for (int u = 0; u < C::OUT; ++u) {
        const int e = tid + u * kThreads, i = e / NS, sl = e % NS;
        if (i < k && s0 + sl < n) X[(int64_t)i * ld + s0 + sl] = out[u];
      }
      continue;
    }
    for (int e = warp; e < C::TILES; e += kWarps) {
      const int mt = e % C::MT, nt = e / C::MT;
      float acc[oz::kSlices][4];
      oz::tile<KP / 16>(acc, dT + mt * 16 * LD, LD, KP * LD, dX + nt * 8 * LD, LD, NS * LD);
      const int sl = nt * 8 + 2 * (lane & 3);
      const int64_t s = s0 + sl;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = mt * 16 + (lane >> 2) + 8 * h;
        if (i >= k || s >= n) continue;
        const double y0 = __fma_rn((double)oz::combine(acc, 2 * h), oz::unit(exT[i], exX[sl]), sm[sl]);
        const double y1 = __fma_rn((double)oz::combine(acc, 2 * h + 1), oz::unit(exT[i], exX[sl + 1]), sm[sl + 1]);
        double* q = X + (int64_t)i * ld + s;
        if (pair_ok && s + 1 < n) {
          *reinterpret_cast<double2*>(q) = make_double2(y0, y1);
        } else {
          q[0] = y0;
          if (s + 1 < n) q[1] = y1;
        }
      }
    }
  }
}

template <int KP>
cudaError_t run_update(double* X, int64_t ld, int64_t n, int k, const double* mean, const double* T, int num_sms,
                       cudaStream_t s) {
  constexpr size_t smem = UpdCfg<KP>::BYTES;
  static_assert(smem <= 227 * 1024, "a CTA's shared memory");
  constexpr int per_sm = std::max(1, std::min<int>(4, 227 * 1024 / (smem + 1024)));
  const cudaError_t e = cudaFuncSetAttribute(update_kernel<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int64_t ntiles = (n + UpdCfg<KP>::NS - 1) / UpdCfg<KP>::NS;
  const int64_t grid = std::min<int64_t>(ntiles, (int64_t)per_sm * num_sms);
  update_kernel<KP><<<(unsigned)grid, kThreads, smem, s>>>(X, ld, n, k, mean, T);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace

namespace mg {

// Two CTAs per SM at most, all with the same number of chunks but the last.
int obs_blocks(int64_t p, int num_sms) {
  const int64_t chunks = std::max<int64_t>(1, (p + kObs - 1) / kObs);
  const int64_t per = (chunks + 2 * (int64_t)num_sms - 1) / (2 * (int64_t)num_sms);
  return (int)((chunks + per - 1) / per);
}

// States up to which the mean rides along: more would run at the products'
// occupancy (their shared memory), not at the copy rate.
bool mean_rides_along(int64_t n) { return n <= 16384; }

cudaError_t launch_obs_products(const ObsProducts& a, cudaStream_t s) {
  const int mean_blocks = a.mean ? (int)((a.n + 255) / 256) : 0;
  return a.eps ? obs_by_k<true>(a, mean_blocks, s) : obs_by_k<false>(a, mean_blocks, s);
}

cudaError_t launch_reduce_parts(const double* part, int nblk, int64_t len, double* out, cudaStream_t s) {
  reduce_parts_kernel<<<(unsigned)((len + 31) / 32), kThreads, 0, s>>>(part, nblk, len, out);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

cudaError_t launch_update_fp64(double* X, int64_t ld, int64_t n, int k, const double* mean, const double* T,
                               int num_sms, cudaStream_t s) {
  if (k <= 16) return run_update<16>(X, ld, n, k, mean, T, num_sms, s);
  if (k <= 32) return run_update<32>(X, ld, n, k, mean, T, num_sms, s);
  if (k <= 48) return run_update<48>(X, ld, n, k, mean, T, num_sms, s);
  if (k <= 64) return run_update<64>(X, ld, n, k, mean, T, num_sms, s);
  if (k <= 96) return run_update<96>(X, ld, n, k, mean, T, num_sms, s);
  return run_update<112>(X, ld, n, k, mean, T, num_sms, s);
}

}  // namespace mg
