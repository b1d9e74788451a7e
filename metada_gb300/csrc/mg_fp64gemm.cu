// FP64 contractions of the global analyses (ETKF.hpp:150-179, EnKF.hpp:180-225)
// on the tensor cores (mg_ozaki.cuh): the obs-space products
//   C = U^T diag(1/sigma^2) V,  b = U^T diag(1/sigma^2) d   (p x k operands)
// and the state update Xa = xm 1^T + X' T (n x k).
#include <algorithm>

#include "mg_internal.h"
#include "mg_ozaki.cuh"

namespace {

namespace oz = mg::oz;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kObs = 64;          // obs per chunk (the contraction of one tile)
constexpr int kLdo = kObs + 8;    // its row stride in halves: 16-byte rows, conflict-free ldmatrix

// ---------------------------------------------------------- cross products --
// Obs chunks of a contiguous range per CTA.  Rows are whitened by 1/sigma
// (one FP64 multiplication per entry), each column gets its own scale, and a
// 16 x 8 tile's integer sum over the chunk is added to the FP64 accumulator
// its lanes keep for the CTA's whole range (two FP64 operations per entry
// and chunk, against 64 multiply-adds).  SYM: V = U, the tiles that touch the
// lower triangle; the innovation is one more column of V.
//
// What the scaled integers cannot hold (non-finite values, magnitudes past
// 2^478, a negative sigma^2) is summed by the plain FP64 loop, chunk by chunk.
// 500,000 obs x 64 members: 4.52 ms (the FP64 units) -> 0.37 ms for the
// symmetric product, 4.39 -> 0.76 ms for the other.
template <int KP, bool SYM>
struct CrossCfg {
  static constexpr int NT = KP / 8 + (SYM ? 1 : 0);     // column tiles of V
  static constexpr int MT = KP / 16;
  static constexpr int TILES = SYM ? MT * (MT + 1) + MT : MT * NT;
  static constexpr int TPW = (TILES + kWarps - 1) / kWarps;
  static constexpr int VROWS = SYM ? 8 : KP;             // digit rows kept for V beside U's
  static constexpr size_t BYTES = sizeof(__half) * oz::kSlices * (KP + VROWS) * kLdo + sizeof(double) * kObs * 2 +
                                  sizeof(int) * (2 * KP + 8 + 4);
};

template <int KP, bool SYM>
__global__ void __launch_bounds__(kThreads) cross_kernel(const double* __restrict__ U, const double* __restrict__ V,
                                                         const double* __restrict__ rinv,
                                                         const double* __restrict__ dinn, int64_t p, int k,
                                                         int64_t per_block, double* __restrict__ part) {
  using C = CrossCfg<KP, SYM>;
  constexpr int SU = KP * kLdo, SV = C::VROWS * kLdo;  // slice strides
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __half* dU = reinterpret_cast<__half*>(smem_raw);
  __half* dV = dU + oz::kSlices * SU;
  double* sw = reinterpret_cast<double*>(dV + oz::kSlices * SV);  // 1/sigma
  double* sd = sw + kObs;                                         // d/sigma (SYM)
  int* exU = reinterpret_cast<int*>(sd + kObs);
  int* exV = exU + KP;  // SYM: one entry, the innovation's
  int* odd = exV + KP + 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t o0 = (int64_t)blockIdx.x * per_block, o1 = min(p, o0 + per_block);
  // The warp's tiles: (row tile, column tile); SYM: column tile MT * 2 is the innovation.
  int tm[C::TPW], tn[C::TPW];
#pragma unroll
  for (int u = 0; u < C::TPW; ++u) {
    int e = warp + u * kWarps;
    tm[u] = -1;
    tn[u] = 0;
    if (e >= C::TILES) continue;
    if (SYM) {
      int m = 0;
      while (e >= 2 * (m + 1) + 1) e -= 2 * (m + 1) + 1, ++m;
      tm[u] = m;
      tn[u] = e < 2 * (m + 1) ? e : 2 * C::MT;
    } else {
      tm[u] = e / C::NT;
      tn[u] = e % C::NT;
    }
  }
  double c64[C::TPW][4];
#pragma unroll
  for (int u = 0; u < C::TPW; ++u)
#pragma unroll
    for (int e = 0; e < 4; ++e) c64[u][e] = 0.0;

  auto digits = [&](const double* A, __half* dst, int* ex, int64_t c0) {
    // items (column, eight obs): whiten, column exponents, then the digits
    constexpr int ITEMS = KP * (kObs / 8), PER = (ITEMS + kThreads - 1) / kThreads;
    double v[PER][8];
#pragma unroll
    for (int x = 0; x < PER; ++x) {
      const int it = tid + x * kThreads;
      const int i = it % KP, og = it / KP;
      int ef = 1;
      if (it < ITEMS) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int64_t o = c0 + og * 8 + q;
          v[x][q] = (i < k && o < o1) ? A[o * k + i] * sw[og * 8 + q] : 0.0;
          ef = max(ef, oz::ef_of(v[x][q]));
        }
        atomicMax(&ex[i], ef);
      }
    }
    __syncthreads();
#pragma unroll
    for (int x = 0; x < PER; ++x) {
      const int it = tid + x * kThreads;
      const int i = it % KP, og = it / KP;
      if (it < ITEMS) {
        const int ef = ex[i];
        if (ef > oz::kMaxEf) *odd = 1;
        oz::store_digits8(v[x], ef, dst + i * kLdo + og * 8, KP * kLdo);
      }
    }
  };

  for (int64_t c0 = o0; c0 < o1; c0 += kObs) {
    for (int i = tid; i < 2 * KP + 8; i += kThreads) exU[i] = 1;
    if (tid == 0) *odd = 0;
    __syncthreads();
    if (tid < kObs) {
      const int64_t o = c0 + tid;
      const double w = o < o1 ? rinv[o] : 0.0;
      if (w < 0.0 || oz::ef_of(w) > oz::kMaxEf) *odd = 1;
      const double s = sqrt(fabs(w));
      sw[tid] = s;
      if (SYM) {
        const double d = o < o1 ? dinn[o] * s : 0.0;
        sd[tid] = d;
        atomicMax(&exV[0], oz::ef_of(d));
      }
    }
    __syncthreads();
    digits(U, dU, exU, c0);
    if (SYM) {
      if (tid < 64) {  // eight columns, the innovation in the first
        const int i = tid & 7, og = tid >> 3;
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = i == 0 ? sd[og * 8 + q] : 0.0;
        const int ef = exV[0];
        if (ef > oz::kMaxEf) *odd = 1;
        oz::store_digits8(v, ef, dV + i * kLdo + og * 8, SV);
      }
    } else {
      digits(V, dV, exV, c0);
    }
    __syncthreads();
    if (*odd) {
      for (int u = 0; u < C::TPW; ++u) {
        if (tm[u] < 0) continue;
        const bool dcol = SYM && tn[u] == 2 * C::MT;
        for (int e = 0; e < 4; ++e) {
          const int i = tm[u] * 16 + (lane >> 2) + 8 * (e >> 1), j = (dcol ? 0 : tn[u] * 8) + 2 * (lane & 3) + (e & 1);
          if (i >= k || j >= (dcol ? 1 : k)) continue;
          double t = 0.0;
          for (int64_t o = c0; o < min(o1, c0 + (int64_t)kObs); ++o)
            t += (U[o * k + i] * rinv[o]) * (dcol ? dinn[o] : (SYM ? U : V)[o * k + j]);
          // tm, tn and c64 stay in registers: select the tile statically
#pragma unroll
          for (int x = 0; x < C::TPW; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y)
              if (x == u && y == e) c64[x][y] += t;
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < C::TPW; ++u) {
        if (tm[u] < 0) continue;
        const bool dcol = SYM && tn[u] == 2 * C::MT;
        const __half* b = SYM ? (dcol ? dV : dU + tn[u] * 8 * kLdo) : dV + tn[u] * 8 * kLdo;
        float acc[oz::kSlices][4];
        oz::tile<kObs / 16>(acc, dU + tm[u] * 16 * kLdo, kLdo, SU, b, kLdo, (SYM && !dcol) ? SU : SV);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = tm[u] * 16 + (lane >> 2) + 8 * (e >> 1), jl = 2 * (lane & 3) + (e & 1);
          const int ev = SYM ? (dcol ? exV[0] : exU[tn[u] * 8 + jl]) : exV[tn[u] * 8 + jl];
          c64[u][e] = __fma_rn((double)oz::combine(acc, e), oz::unit(exU[i], ev), c64[u][e]);
        }
      }
    }
    __syncthreads();
  }
  double* out = part + (size_t)blockIdx.x * (k * k + (SYM ? k : 0));
#pragma unroll
  for (int u = 0; u < C::TPW; ++u) {
    if (tm[u] < 0) continue;
    const bool dcol = SYM && tn[u] == 2 * C::MT;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = tm[u] * 16 + (lane >> 2) + 8 * (e >> 1), jl = 2 * (lane & 3) + (e & 1);
      if (i >= k) continue;
      if (dcol) {
        if (jl == 0) out[k * k + i] = c64[u][e];
        continue;
      }
      const int j = tn[u] * 8 + jl;
      if (j >= k || (SYM && j > i)) continue;
      out[i * k + j] = c64[u][e];
      if (SYM) out[j * k + i] = c64[u][e];
    }
  }
}

template <int KP, bool SYM>
cudaError_t run_cross(const double* U, const double* V, const double* rinv, const double* dinn, int64_t p, int k,
                      int nblk, int64_t per_block, double* part, cudaStream_t s) {
  const size_t smem = CrossCfg<KP, SYM>::BYTES;
  const cudaError_t e =
      cudaFuncSetAttribute(cross_kernel<KP, SYM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  cross_kernel<KP, SYM><<<nblk, kThreads, smem, s>>>(U, V, rinv, dinn, p, k, per_block, part);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

template <bool SYM>
cudaError_t cross(const double* U, const double* V, const double* rinv, const double* dinn, int64_t p, int k, int nblk,
                  double* part, cudaStream_t s) {
  const int64_t chunks = (p + kObs - 1) / kObs, per_block = (chunks + nblk - 1) / nblk * kObs;
  if (k <= 16) return run_cross<16, SYM>(U, V, rinv, dinn, p, k, nblk, per_block, part, s);
  if (k <= 32) return run_cross<32, SYM>(U, V, rinv, dinn, p, k, nblk, per_block, part, s);
  if (k <= 64) return run_cross<64, SYM>(U, V, rinv, dinn, p, k, nblk, per_block, part, s);
  return run_cross<112, SYM>(U, V, rinv, dinn, p, k, nblk, per_block, part, s);
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
  int* odd = exX + NS;  // [0]: this tile, [1]: T
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < KP; i += kThreads) exT[i] = 1;
  if (tid < 2) odd[tid] = 0;
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
    oz::store_digits8(v, exT[i], dT + i * LD + jg * 8, KP * LD);
  }
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
      if (ef > oz::kMaxEf) odd[0] = 1;
      oz::store_digits8(v[x], ef, dX + sl * LD + jg * 8, NS * LD);
    }
    __syncthreads();
    if (odd[0]) {  // magnitudes the integers cannot hold: the plain FP64 sum
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
  const size_t smem = UpdCfg<KP>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(update_kernel<KP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, update_kernel<KP>, kThreads, smem);
  if (e != cudaSuccess) return e;
  const int64_t ntiles = (n + UpdCfg<KP>::NS - 1) / UpdCfg<KP>::NS;
  const int64_t grid = std::min<int64_t>(ntiles, (int64_t)std::max(per_sm, 1) * num_sms);
  update_kernel<KP><<<(unsigned)grid, kThreads, smem, s>>>(X, ld, n, k, mean, T);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace

namespace mg {

// Two CTAs per SM at most, all with the same number of chunks but the last.
int cross_blocks(int64_t p, int num_sms) {
  const int64_t chunks = std::max<int64_t>(1, (p + kObs - 1) / kObs);
  const int64_t per = (chunks + 2 * (int64_t)num_sms - 1) / (2 * (int64_t)num_sms);
  return (int)((chunks + per - 1) / per);
}

cudaError_t launch_gram_fp64(const double* Y, const double* rinv, const double* dinn, int64_t p, int k, int nblk,
                             double* part, cudaStream_t s) {
  return cross<true>(Y, Y, rinv, dinn, p, k, nblk, part, s);
}

cudaError_t launch_cross_fp64(const double* U, const double* V, const double* rinv, int64_t p, int k, int nblk,
                              double* part, cudaStream_t s) {
  return cross<false>(U, V, rinv, nullptr, p, k, nblk, part, s);
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
