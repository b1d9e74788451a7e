// FP64 local analyses with the symmetric square root (Hunt et al. 2007),
// k <= 96: one CTA of 256 threads per analysis, a persistent grid pulling
// points from a counter in the grid's column order.
//
// Per analysis: the column's candidates are filtered by level and weighted
// in FP64 (the oracle's operation order), the whitened rows of Y' are
// gathered 32 at a time and Y'^T R^-1 Y' and Y'^T R^-1 d accumulated on the
// tensor cores by exact splitting (mg_ozaki.cuh), and the inverse square root
// comes from an FP32 eigenbasis corrected in FP64 (mg_hunt.cuh), in a second
// pass where the system is graded (the CTA keeps it in global memory for that).
// A point whose correction does not apply is handed back (redo list) to the
// FP64 Jacobi kernel.  What bounds it: the FP32 Jacobi's shared-memory rounds and
// the 2.3 k^3 FP64 multiply-adds of the correction, which CTAs of one SM
// overlap (three at k <= 64).  60 x 30 x 10 points, k = 64, about 290 local
// obs: 782 ms with the FP64 Jacobi (ten sweeps on the FP64 units) -> 57 ms.
#include <algorithm>

#include "mg_hunt.cuh"
#include "mg_internal.h"
#include "mg_letkf.cuh"
#include "mg_ozaki.cuh"

namespace {

namespace oz = mg::oz;
using mg::LetkfParams;

constexpr int kThreads = mg::kHuntThreads;
constexpr int kWarps = kThreads / 32;
constexpr int kObs = 32;        // rows per product
constexpr int kLdo = kObs + 8;  // digit row stride in halves
constexpr int kVars = 8;        // variables per update batch

// Gaspari-Cohn in the operation order of mg::gaspari_cohn<double>, the
// divisions by constants as corrected products (same quotients).
__device__ __forceinline__ double gc64(double z) {
  z = fabs(z);
  if (z >= 2.0) return 0.0;
  if (z <= 1.0) return (((-0.25 * z + 0.5) * z + 0.625) * z - (5.0 / 3.0)) * z * z + 1.0;
  return ((((mg::div_refined(z, 12.0, 1.0 / 12.0) - 0.5) * z + 0.625) * z + 5.0 / 3.0) * z - 5.0) * z + 4.0 -
         2.0 / (3.0 * z);
}

// Half of a localisation support as a divisor of div_refined, which needs the
// divisor and its reciprocal normal (1 / inf is zero, and the quotient's
// remainder 0 x inf).  Above 2^800, infinite supports included (no localisation
// in that direction), the quotient of any finite distance rounds to weight 1;
// 0 and NaN stay (no obs).
__device__ __forceinline__ double half_support(double support) {
  const double c = fabs(0.5 * support), big = 0x1p800, small = 0x1p-800;
  return c > big ? big : (c < small && c > 0.0 ? small : c);
}

template <int KP>
struct Cfg {
  using H = mg::Hunt<KP>;
  static constexpr int MT = KP / 16;
  static constexpr int TILES = MT * (MT + 1) + MT;  // lower triangle and the innovation column
  static constexpr int TPW = (TILES + kWarps - 1) / kWarps;
  static constexpr int SU = KP * kLdo, SD = 8 * kLdo;  // digit slice strides
  static constexpr size_t SEL_BYTES = sizeof(int) * 1024 + sizeof(double) * 512;
  static constexpr size_t A_BYTES = (H::A_BYTES > SEL_BYTES ? H::A_BYTES : SEL_BYTES) / 16 * 16 + 16;
  static constexpr size_t DIG_BYTES = sizeof(__half) * oz::kSlices * (SU + SD);
  static constexpr size_t WORK_BYTES = (H::WORK_BYTES > DIG_BYTES ? H::WORK_BYTES : DIG_BYTES) / 16 * 16 + 16;
  static constexpr size_t BYTES = A_BYTES + WORK_BYTES + H::VEC_BYTES + sizeof(double) * 2 * KP +
                                  sizeof(int) * (KP + 24);
  static constexpr int CTAS = KP <= 32 ? 4 : (KP <= 64 ? 3 : 1);
};

template <int KP>
__global__ void __launch_bounds__(kThreads, Cfg<KP>::CTAS) letkf_hunt_kernel(LetkfParams prm) {
  using C = Cfg<KP>;
  using H = mg::Hunt<KP>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* const work = smem_raw + C::A_BYTES;
  H h;
  h.carve(smem_raw, work, work + C::WORK_BYTES);
  double* bvec = reinterpret_cast<double*>(work + C::WORK_BYTES + H::VEC_BYTES);  // KP
  double* pb = bvec + KP;                                                         // KP: A^-1/2 b
  int* exU = reinterpret_cast<int*>(pb + KP);                                     // KP, then the innovation's
  int* odd = exU + KP + 1;
  int* wcnt = odd + 1;  // kWarps
  // selection (before A exists): candidates (obs, entry), 1/sigma-weights
  int* cand_o = reinterpret_cast<int*>(smem_raw);
  int* cand_e = cand_o + 512;
  double* sw = reinterpret_cast<double*>(cand_e + 512);
  double* sd = sw + 256;
  __half* dU = reinterpret_cast<__half*>(work);
  __half* dD = dU + oz::kSlices * C::SU;
  // update rows, in what the transform leaves free
  double* rX = reinterpret_cast<double*>(h.F);
  double* rT = rX + (kVars + 1) * KP;
  double* rY = h.H;
  static_assert(2 * (kVars + 1) * KP * sizeof(double) <= H::F_BYTES + H::BLK_BYTES, "update rows");
  static_assert((kVars + 1) * KP * sizeof(double) <= H::B_BYTES, "update rows");
  __shared__ long long s_item;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = prm.k;
  const double* Y = static_cast<const double*>(prm.Y);
  const double* Xp = static_cast<const double*>(prm.Xp);
  const bool r_identity = prm.flags & MG_R_IDENTITY;
  const bool infl_compat = prm.flags & MG_INFL_COMPAT;
  const bool upd_compat = prm.flags & MG_UPDATE_COMPAT;
  const bool rtps = prm.flags & MG_RTPS;
  const double hc = half_support(prm.hsupport), vc = half_support(prm.vsupport), vs = prm.vsupport;
  const double rhc = 1.0 / hc, rvc = 1.0 / vc;
  const double diag = (infl_compat || rtps) ? (double)(k - 1) : (double)(k - 1) / prm.rho;
  const double sc = infl_compat ? prm.rho : 1.0;
  const double cw = sqrt((double)(k - 1) * sc);
  int tm[C::TPW], tn[C::TPW];  // the warp's product tiles; column tile 2 MT: the innovation
#pragma unroll
  for (int u = 0; u < C::TPW; ++u) {
    int e = warp + u * kWarps, m = 0;
    tm[u] = -1;
    tn[u] = 0;
    if (e >= C::TILES) continue;
    while (e >= 2 * (m + 1) + 1) e -= 2 * (m + 1) + 1, ++m;
    tm[u] = m;
    tn[u] = e < 2 * (m + 1) ? e : 2 * C::MT;
  }

  for (;;) {
    if (tid == 0) s_item = (long long)atomicAdd(prm.next, 1ull);
    __syncthreads();
    const long long item = s_item;
    __syncthreads();
    if (item >= prm.npoints) break;
    const int lev = (int)(item % prm.nlev);
    const int64_t col = item / prm.nlev;
    const int64_t base = prm.col_base[col] + (int64_t)lev * prm.lev_stride;
    const int64_t e0 = prm.loc_off[col], e1 = prm.loc_off[col + 1];
    double c64[C::TPW][4];
#pragma unroll
    for (int u = 0; u < C::TPW; ++u)
#pragma unroll
      for (int e = 0; e < 4; ++e) c64[u][e] = 0.0;

    // Weights of nb (<= 256) candidates and their products.
    auto batch = [&](int nb) {
      double w = 0.0;
      int o = 0;
      if (tid < nb) {
        o = cand_o[tid];
        const int64_t e = e0 + cand_e[tid];
        w = 1.0;
        if (!r_identity) {
          if (prm.obs_lev) w *= gc64(mg::div_refined(fabs((double)lev - prm.obs_lev[o]), vc, rvc));
          if (prm.loc_dist) w *= gc64(mg::div_refined(prm.loc_dist[e], hc, rhc));
          w *= prm.rinv[o];
          if (!(w > 0.0)) w = 0.0;
        }
      }
      const double s = sqrt(w);
      sw[tid] = s;
      sd[tid] = w > 0.0 ? prm.dinn[o] * s : 0.0;
      const int kept = __syncthreads_count(w > 0.0);
      for (int r0 = 0; r0 < nb; r0 += kObs) {
        for (int i = tid; i < KP + 2; i += kThreads) exU[i] = i == KP + 1 ? 0 : 1;  // exponents, then odd
        __syncthreads();
        constexpr int ITEMS = KP * (kObs / 8), PER = (ITEMS + kThreads - 1) / kThreads;
        double v[PER][8];
#pragma unroll
        for (int x = 0; x < PER; ++x) {
          const int it = tid + x * kThreads, i = it % KP, og = it / KP;
          if (it >= ITEMS) continue;
          int ef = 1;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int r = r0 + og * 8 + q;
            v[x][q] = (i < k && r < nb && sw[r] != 0.0) ? Y[(int64_t)cand_o[r] * k + i] * sw[r] : 0.0;
            ef = max(ef, oz::ef_of(v[x][q]));
          }
          atomicMax(&exU[i], ef);
        }
        if (tid < kObs) atomicMax(&exU[KP], oz::ef_of(r0 + tid < nb ? sd[r0 + tid] : 0.0));
        __syncthreads();
#pragma unroll
        for (int x = 0; x < PER; ++x) {
          const int it = tid + x * kThreads, i = it % KP, og = it / KP;
          if (it >= ITEMS) continue;
          if (exU[i] > oz::kMaxEf) *odd = 1;
          oz::store_digits8(v[x], exU[i], dU + i * kLdo + og * 8, C::SU);
        }
        if (tid < 32) {
          const int i = tid & 7, og = tid >> 3;
          double x[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) x[q] = (i == 0 && r0 + og * 8 + q < nb) ? sd[r0 + og * 8 + q] : 0.0;
          if (exU[KP] > oz::kMaxEf) *odd = 1;
          oz::store_digits8(x, exU[KP], dD + i * kLdo + og * 8, C::SD);
        }
        __syncthreads();
        const bool plain = *odd != 0;  // not finite or out of range: the FP64 sum
#pragma unroll
        for (int u = 0; u < C::TPW; ++u) {
          if (tm[u] < 0) continue;
          const bool dcol = tn[u] == 2 * C::MT;
          float acc[oz::kSlices][4];
          if (!plain)
            oz::tile<kObs / 16>(acc, dU + tm[u] * 16 * kLdo, kLdo, C::SU, dcol ? dD : dU + tn[u] * 8 * kLdo, kLdo,
                                dcol ? C::SD : C::SU);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = tm[u] * 16 + (lane >> 2) + 8 * (e >> 1), jl = 2 * (lane & 3) + (e & 1);
            if (!plain) {
              const int ev = exU[dcol ? KP : tn[u] * 8 + jl];
              c64[u][e] = __fma_rn((double)oz::combine(acc, e), oz::unit(exU[i], ev), c64[u][e]);
            } else {
              const int j = tn[u] * 8 + jl;
              if (i >= k || (dcol ? jl > 0 : j >= k)) continue;
              for (int r = r0; r < min(nb, r0 + kObs); ++r) {
                if (sw[r] == 0.0) continue;
                const double* y = Y + (int64_t)cand_o[r] * k;
                c64[u][e] += (y[i] * sw[r]) * (dcol ? sd[r] : y[j] * sw[r]);
              }
            }
          }
        }
        __syncthreads();
      }
      return kept;
    };

    int nc = 0, nloc = 0;
    for (int64_t c0 = e0; c0 < e1; c0 += kThreads) {
      bool keep = c0 + tid < e1;
      int o = 0;
      if (keep) {
        o = prm.loc_idx[c0 + tid];
        if (prm.obs_lev) keep = !(fabs((double)lev - prm.obs_lev[o]) > vs);
      }
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      if (lane == 0) wcnt[warp] = __popc(bal);
      __syncthreads();
      int pos = nc + __popc(bal & ((1u << lane) - 1u));
#pragma unroll
      for (int q = 0; q < kWarps; ++q) {
        if (q < warp) pos += wcnt[q];
        nc += wcnt[q];
      }
      if (keep) {
        cand_o[pos] = o;
        cand_e[pos] = (int)(c0 + tid - e0);
      }
      __syncthreads();
      if (nc >= kThreads) {
        nloc += batch(kThreads);
        nc -= kThreads;
        const int mo = tid < nc ? cand_o[kThreads + tid] : 0, me = tid < nc ? cand_e[kThreads + tid] : 0;
        __syncthreads();
        cand_o[tid] = mo;
        cand_e[tid] = me;
        __syncthreads();
      }
    }
    if (nc > 0) nloc += batch(nc);

    if (nloc == 0) {
      // LETKF.hpp:167-190: no local obs, x' *= sqrt(rho) (RTPS: unchanged).
      const double sr = rtps ? 1.0 : sqrt(prm.rho);
      for (int e = tid; e < prm.n_var * k; e += kThreads) {
        const int v = e / k, i = e - v * k;
        const int64_t s = base + (int64_t)v * prm.var_stride;
        mg::letkf_store(prm, s * k + i, prm.xmean[s] + Xp[s * k + i] * sr);
      }
      if (tid == 0) atomicAdd(prm.n_empty, 1ull);
      __syncthreads();
      continue;
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < C::TPW; ++u) {
      if (tm[u] < 0) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = tm[u] * 16 + (lane >> 2) + 8 * (e >> 1), jl = 2 * (lane & 3) + (e & 1);
        const int j = tn[u] * 8 + jl;
        if (i >= k) continue;
        if (tn[u] == 2 * C::MT) {
          if (jl == 0) bvec[i] = c64[u][e];
        } else if (j <= i) {
          h.A[mg::tri(i, j)] = c64[u][e] + (i == j ? diag : 0.0);
        }
      }
    }
    __syncthreads();
    const int npack = k * (k + 1) / 2;
    for (int e = tid; e < npack; e += kThreads) prm.gram[(size_t)blockIdx.x * H::PACKED + e] = h.A[e];
    double scale;
    int sweeps = 0;
    auto reload = [&] {  // each thread what it wrote
      for (int e = tid; e < npack; e += kThreads) h.A[e] = prm.gram[(size_t)blockIdx.x * H::PACKED + e];
    };
    if (!h.template transform<false>(k, diag, &scale, &sweeps, reload)) {
      if (tid == 0) prm.redo_out[atomicAdd(prm.n_redo, 1ull)] = (int32_t)(col * prm.nlev + lev);
      __syncthreads();
      continue;
    }

    if (upd_compat) {  // per-member update, LETKF.hpp:232-238: wa = sc M (M b), row sums of W = cw M 1
      for (int i = tid; i < k; i += kThreads) {
        rX[i] = bvec[i];
        rX[KP + i] = 1.0;
      }
      __syncthreads();
      h.apply(rX, rT, rY, 2, k);
      for (int i = tid; i < k; i += kThreads) {
        pb[i] = cw * scale * rY[KP + i];
        rX[i] = rY[i];
      }
      __syncthreads();
      h.apply(rX, rT, rY, 1, k);
      for (int e = tid; e < prm.n_var * k; e += kThreads) {
        const int v = e / k, i = e - v * k;
        const int64_t s = base + (int64_t)v * prm.var_stride;
        const double xp = Xp[s * k + i];
        mg::letkf_store(prm, s * k + i, (prm.xmean[s] + xp * (sc * scale * scale * rY[i])) + xp * pb[i]);
      }
    } else {  // xa = xm + x'.wa + W x', with M = A^-1/2: x'.wa = sc (M x').(M b), W x' = cw M x'
      for (int v0 = 0; v0 < prm.n_var; v0 += kVars) {
        const int nv = min(kVars, prm.n_var - v0);
        for (int e = tid; e < nv * k; e += kThreads) {
          const int v = e / k, i = e - v * k;
          rX[v * KP + i] = Xp[(base + (int64_t)(v0 + v) * prm.var_stride) * k + i];
        }
        if (v0 == 0)
          for (int i = tid; i < k; i += kThreads) rX[nv * KP + i] = bvec[i];
        __syncthreads();
        h.apply(rX, rT, rY, nv + (v0 == 0), k);
        if (v0 == 0) {
          for (int i = tid; i < k; i += kThreads) pb[i] = rY[nv * KP + i];
          __syncthreads();
        }
        if (warp < nv) {  // one warp per variable
          const int64_t s = base + (int64_t)(v0 + warp) * prm.var_stride;
          const double* y = rY + warp * KP;
          double inc = 0.0, sb = 0.0, sa = 0.0;
          for (int i = lane; i < k; i += 32) {
            inc = __fma_rn(y[i], pb[i], inc);
            if (rtps) {
              const double xb = Xp[s * k + i];
              sb = __fma_rn(xb, xb, sb);
              sa = __fma_rn(y[i], y[i], sa);
            }
          }
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) {
            inc += __shfl_xor_sync(0xffffffffu, inc, off);
            sb += __shfl_xor_sync(0xffffffffu, sb, off);
            sa += __shfl_xor_sync(0xffffffffu, sa, off);
          }
          const double g = cw * scale;
          double f = 0.0;  // relaxation to prior spread: factor - 1
          if (rtps) {
            sb = sqrt(sb / (k - 1));
            sa = g * sqrt(sa / (k - 1));
            f = (sa > 0.0) ? prm.rho * (sb - sa) / sa : 0.0;
          }
          const double xi = prm.xmean[s] + sc * scale * scale * inc;
          for (int i = lane; i < k; i += 32) {
            const double s2 = g * y[i];
            mg::letkf_store(prm, s * k + i, (xi + s2) + f * s2);
          }
        }
        __syncthreads();
      }
    }
    if (tid == 0) {
      atomicAdd(prm.total_local, (unsigned long long)nloc);
      atomicAdd(prm.total_sweeps, (unsigned long long)sweeps);
      atomicMax(prm.max_local, nloc);
      atomicMax(prm.max_sweeps, sweeps);
    }
    __syncthreads();
  }
}

template <int KP>
cudaError_t launch(const LetkfParams& prm, int num_sms, cudaStream_t s) {
  const size_t smem = Cfg<KP>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(letkf_hunt_kernel<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, letkf_hunt_kernel<KP>, kThreads, smem);
  if (e != cudaSuccess) return e;
  per_sm = std::max(1, std::min(per_sm, Cfg<KP>::CTAS));  // prm.gram has a system for each
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)per_sm * num_sms, prm.npoints));
  letkf_hunt_kernel<KP><<<(unsigned)grid, kThreads, smem, s>>>(prm);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

// ------------------------------------------------------------ global ETKF --
// The same transform of one system: a CTA factors it and leaves V and Ws;
// rows of T = (wa_j + W_ji) follow on as many CTAs as there are rows / 8.
// k = 64: 5.69 ms by FP64 Jacobi -> 0.55 + 0.04 ms.
template <int KP>
__global__ void __launch_bounds__(kThreads) hunt_factor_kernel(const double* __restrict__ Gb, int k, double diag,
                                                               float* __restrict__ Vout, double* __restrict__ Wout,
                                                               double* __restrict__ info) {
  using H = mg::Hunt<KP>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr size_t AB = (H::A_BYTES + 15) / 16 * 16;
  H h;
  h.carve(smem_raw, smem_raw + AB, smem_raw + AB + (H::WORK_BYTES + 15) / 16 * 16);
  const int tid = threadIdx.x;
  auto load = [&] {
    for (int e = tid; e < k * k; e += kThreads) {
      const int i = e / k, j = e - i * k;
      if (j <= i) h.A[mg::tri(i, j)] = Gb[e] + (i == j ? diag : 0.0);
    }
  };
  load();
  __syncthreads();
  double scale = 0.0;
  int sweeps = 0;
  const bool ok = h.template transform<(KP <= 64)>(k, diag, &scale, &sweeps, load);
  if (tid == 0) info[0] = ok ? scale : 0.0;
  if (!ok) return;
  for (int e = tid; e < k * H::LDV; e += kThreads) Vout[e] = h.V[e];
  for (int e = tid; e < k * (k + 1) / 2; e += kThreads) Wout[e] = h.A[e];
}

template <int KP>
__global__ void __launch_bounds__(kThreads) hunt_rows_kernel(const double* __restrict__ Gb, int k, double out_scale,
                                                             const float* __restrict__ Vin,
                                                             const double* __restrict__ Win,
                                                             const double* __restrict__ info, double* __restrict__ T) {
  using H = mg::Hunt<KP>;
  constexpr int ROWS = 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  H h;
  h.V = reinterpret_cast<float*>(smem_raw);
  h.A = reinterpret_cast<double*>(smem_raw + (H::V_BYTES + 15) / 16 * 16);
  double* rX = h.A + H::PACKED;
  double* rT = rX + (ROWS + 1) * KP;
  double* rY = rT + (ROWS + 1) * KP;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double scale = info[0];
  if (scale == 0.0) return;  // the FP64 Jacobi solves this one
  const int r0 = blockIdx.x * ROWS, nr = min(ROWS, k - r0);
  for (int e = tid; e < k * H::LDV; e += kThreads) h.V[e] = Vin[e];
  for (int e = tid; e < k * (k + 1) / 2; e += kThreads) h.A[e] = Win[e];
  for (int e = tid; e < (nr + 1) * k; e += kThreads) {
    const int r = e / k, i = e - r * k;
    rX[r * KP + i] = r < nr ? (i == r0 + r ? 1.0 : 0.0) : Gb[k * k + i];
  }
  __syncthreads();
  h.apply(rX, rT, rY, nr + 1, k);
  if (warp >= nr) return;
  const double *y = rY + warp * KP, *yb = rY + nr * KP;
  double wa = 0.0;
  for (int i = lane; i < k; i += 32) wa = __fma_rn(y[i], yb[i], wa);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) wa += __shfl_xor_sync(0xffffffffu, wa, off);
  const double g = sqrt((double)(k - 1)) * scale;
  for (int i = lane; i < k; i += 32) T[(r0 + warp) * k + i] = out_scale * (scale * scale * wa + g * y[i]);
}

template <int KP>
cudaError_t solve_global(const double* Gb, int k, double diag, double out_scale, void* ws, double* T, cudaStream_t s) {
  using H = mg::Hunt<KP>;
  float* V = static_cast<float*>(ws);
  double* W = reinterpret_cast<double*>(V + KP * H::LDV);
  double* info = W + H::PACKED;
  const size_t sf = (H::A_BYTES + 15) / 16 * 16 + (H::WORK_BYTES + 15) / 16 * 16 + H::VEC_BYTES;
  const size_t sr = (H::V_BYTES + 15) / 16 * 16 + sizeof(double) * (H::PACKED + 27 * KP);
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(hunt_factor_kernel<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sf)) !=
          cudaSuccess ||
      (e = cudaFuncSetAttribute(hunt_rows_kernel<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sr)) !=
          cudaSuccess)
    return e;
  hunt_factor_kernel<KP><<<1, kThreads, sf, s>>>(Gb, k, diag, V, W, info);
  MG_COUNT_LAUNCH();
  hunt_rows_kernel<KP><<<(k + 7) / 8, kThreads, sr, s>>>(Gb, k, out_scale, V, W, info, T);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

template <int KP>
constexpr size_t global_bytes() {
  using H = mg::Hunt<KP>;
  return sizeof(float) * KP * H::LDV + sizeof(double) * (H::PACKED + 1);
}

}  // namespace

namespace mg {

cudaError_t letkf_hunt_launch(const LetkfParams& prm, int num_sms, cudaStream_t s) {
  if (prm.k <= 32) return launch<32>(prm, num_sms, s);
  if (prm.k <= 64) return launch<64>(prm, num_sms, s);
  return launch<96>(prm, num_sms, s);
}

size_t letkf_hunt_doubles(int k, int num_sms) {
  const size_t per_sm = k <= 32 ? Cfg<32>::CTAS * Hunt<32>::PACKED
                                : (k <= 64 ? Cfg<64>::CTAS * Hunt<64>::PACKED : Cfg<96>::CTAS * Hunt<96>::PACKED);
  return per_sm * num_sms;
}

size_t hunt_global_bytes(int k) {
  return k <= 32 ? global_bytes<32>() : (k <= 64 ? global_bytes<64>() : global_bytes<112>());
}

const double* hunt_global_info(const void* ws, int k) {
  return reinterpret_cast<const double*>(static_cast<const char*>(ws) + hunt_global_bytes(k)) - 1;
}

cudaError_t launch_hunt_global(const double* Gb, int k, double diag, double out_scale, void* ws, double* T,
                               cudaStream_t s) {
  if (k <= 32) return solve_global<32>(Gb, k, diag, out_scale, ws, T, s);
  if (k <= 64) return solve_global<64>(Gb, k, diag, out_scale, ws, T, s);
  return solve_global<112>(Gb, k, diag, out_scale, ws, T, s);
}

}  // namespace mg
