// FP64 local analyses with the reference's Cholesky square root
// (LETKF.hpp:214-238, flags with MG_SQRT_CHOLESKY).
//
// The reference inverts A = (k-1) I + Y'^T R^-1 Y' and takes the lower
// Cholesky factor of Pa = A^-1.  With the factorisation from the last index
// up, A = U D U^T (U unit upper triangular), Pa = (U^-T D^-1/2)(U^-T D^-1/2)^T
// with a lower triangular factor of positive diagonal, so chol_L(Pa) =
// U^-T D^-1/2 =: M by uniqueness: no inverse and no second factorisation.
// What the update needs from it are triangular solves:
//   wa = Pa b       = U^-T D^-1 U^-1 b,
//   row sums of M   = U^-T D^-1/2 1          (per-member scalar update),
//   M^T x           = D^-1/2 U^-1 x          (X' W update).
//
// GB300 runs two FP64 lanes per clock per SM, so a warp instruction takes
// its scheduler's FP64 unit 64 cycles, whatever the lanes hold: the kernel is
// laid out for few FP64 warp instructions and no idle lanes.  One analysis
// belongs to a group of one warp (k <= 32) or four warps (k <= 96, and fewer
// members where the points are few), its threads a TI x TJ grid of interleaved register tiles of A's lower triangle
// (tiles above the diagonal are not formed), several groups per SM covering
// each other's latencies.  The root-free factorisation needs one reciprocal
// per column, from an FP32 seed and one third-order Newton step (three FP64
// instructions); the square roots are taken for all columns at once.
// Measured on a 144 x 72 grid, k = 32, 28 local obs: 5.33 ms (one CTA per
// point, inverse and two Cholesky factorisations with a barrier per column)
// -> 0.64 ms.
#include <algorithm>

#include "mg_fp64.cuh"
#include "mg_internal.h"
#include "mg_letkf.cuh"

namespace {

using mg::LetkfParams;
using mg::gaspari_cohn;

constexpr int kThreads = 128;

template <int KMAX, int NW>  // NW: warps per analysis
struct Cfg {
  static constexpr int TI = NW == 1 ? 8 : 16, TJ = TI / 2;  // thread grid
  static constexpr int RA = KMAX / TI;                 // tile rows; tile columns of row a: 2 (a + 1)
  static constexpr int NT = RA * (RA + 1);             // tiles of the lower triangle
  static constexpr int NV = KMAX <= 32 ? 1 : KMAX / 32;  // vector elements per lane
  static constexpr int GROUPS = kThreads / (32 * NW);  // analyses per CTA
  static constexpr int LDS = KMAX + 1;
  static constexpr int SEL = 32 * NW;                  // list entries filtered at a time
  static constexpr int CH = 16;                        // rows gathered at a time
  // doubles: factor, gathered rows, row buffers, selected weights and
  // weighted innovations, 1/d, d, wa, row sums; then selected obs
  static constexpr int DOUBLES = KMAX * LDS + CH * KMAX + 2 * KMAX + 2 * SEL + 4 * KMAX;
  static constexpr size_t BYTES = GROUPS * (sizeof(double) * DOUBLES + sizeof(int) * (SEL + 8));
};

template <int KMAX, int NW>
__global__ void __launch_bounds__(kThreads, KMAX <= 64 ? 5 : 2) letkf_chol_kernel(LetkfParams prm) {
  using C = Cfg<KMAX, NW>;
  constexpr int TI = C::TI, TJ = C::TJ, RA = C::RA, NV = C::NV, LDS = C::LDS, SEL = C::SEL, CH = C::CH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  const int gid = threadIdx.x / (32 * NW);          // group in the CTA
  const int t = threadIdx.x - gid * 32 * NW;        // thread in the group
  const int gw = t >> 5;                            // warp in the group
  double* S = reinterpret_cast<double*>(smem_raw) + gid * C::DOUBLES;  // row j: u_l of column j, l < j
  double* Ys = S + KMAX * LDS;
  double* row = Ys + CH * KMAX;   // two buffers
  double* sel_w = row + 2 * KMAX;
  double* sel_sd = sel_w + SEL;
  double* dinv = sel_sd + SEL;
  double* dval = dinv + KMAX;
  double* wa_s = dval + KMAX;
  double* rs_s = wa_s + KMAX;
  int* sel_o = reinterpret_cast<int*>(reinterpret_cast<double*>(smem_raw) + C::GROUPS * C::DOUBLES) + gid * (SEL + 8);
  int* wcnt = sel_o + SEL;  // per-warp counts; [4]: the item
  auto gsync = [] {
    if (NW == 1) __syncwarp();
    else __syncthreads();
  };
  const int li = t / TJ, lj = t % TJ;
  const int k = prm.k;
  const double* Y = static_cast<const double*>(prm.Y);
  const double* Xp = static_cast<const double*>(prm.Xp);
  const bool r_identity = prm.flags & MG_R_IDENTITY;
  const bool infl_compat = prm.flags & MG_INFL_COMPAT;
  const bool upd_compat = prm.flags & MG_UPDATE_COMPAT;
  const bool rtps = prm.flags & MG_RTPS;
  const double hc = 0.5 * prm.hsupport, vc = 0.5 * prm.vsupport, vs = prm.vsupport;
  const double diag = (infl_compat || rtps) ? (double)(k - 1) : (double)(k - 1) / prm.rho;
  const double sc = infl_compat ? prm.rho : 1.0;
  const double cw = sqrt((double)(k - 1) * sc);

  for (;;) {
    long long item;
    if (NW == 1) {
      if (lane == 0) item = (long long)atomicAdd(prm.next, 1ull);
      item = __shfl_sync(0xffffffffu, item, 0);
    } else {
      __shared__ long long s_item;
      if (threadIdx.x == 0) s_item = (long long)atomicAdd(prm.next, 1ull);
      __syncthreads();
      item = s_item;
    }
    if (item >= prm.npoints) break;
    const int lev = (int)(item % prm.nlev);
    const int64_t col = item / prm.nlev;
    const int64_t base = prm.col_base[col] + (int64_t)lev * prm.lev_stride;
    const int64_t e0 = prm.loc_off[col], e1 = prm.loc_off[col + 1];

    // ---- Gram and b = Y'^T R^-1 d (b in the group's first warp) ----
    double acc[C::NT];
#pragma unroll
    for (int u = 0; u < C::NT; ++u) acc[u] = 0.0;
    double bv[NV];
#pragma unroll
    for (int m = 0; m < NV; ++m) bv[m] = 0.0;
    int nloc = 0;
    for (int64_t c0 = e0; c0 < e1; c0 += SEL) {
      bool keep = c0 + t < e1;
      int o = 0;
      double w = 1.0;
      if (keep) {
        o = prm.loc_idx[c0 + t];
        if (prm.obs_lev) {
          const double dl = fabs((double)lev - prm.obs_lev[o]);
          if (dl > vs) keep = false;
          else if (!r_identity) w *= gaspari_cohn<double>(dl / vc);
        }
        if (keep && !r_identity) {
          if (prm.loc_dist) w *= gaspari_cohn<double>(prm.loc_dist[c0 + t] / hc);
          w *= prm.rinv[o];
          if (!(w > 0.0)) keep = false;
        }
      }
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      int pos = __popc(bal & ((1u << lane) - 1u)), cnt = __popc(bal);
      if (NW > 1) {
        if (lane == 0) wcnt[gw] = cnt;
        __syncthreads();
        cnt = 0;
#pragma unroll
        for (int q = 0; q < NW; ++q) {
          if (q < gw) pos += wcnt[q];
          cnt += wcnt[q];
        }
      }
      if (keep) {
        sel_o[pos] = o;
        sel_w[pos] = w;
        sel_sd[pos] = w * prm.dinn[o];
      }
      gsync();
      for (int r0 = 0; r0 < cnt; r0 += CH) {
        const int nr = min(CH, cnt - r0);
        for (int e = t; e < nr * KMAX; e += 32 * NW) {
          const int r = e / KMAX, j = e - r * KMAX;
          Ys[e] = j < k ? Y[(int64_t)sel_o[r0 + r] * k + j] : 0.0;
        }
        gsync();
        for (int r = 0; r < nr; ++r) {
          const double* y = Ys + r * KMAX;
          double av[RA];
#pragma unroll
          for (int a = 0; a < RA; ++a) av[a] = y[TI * a + li];
          if (!r_identity) {
            const double wr = sel_w[r0 + r];
#pragma unroll
            for (int a = 0; a < RA; ++a) av[a] *= wr;
          }
#pragma unroll
          for (int b = 0; b < 2 * RA; ++b) {
            const double yb = y[TJ * b + lj];
#pragma unroll
            for (int a = b / 2; a < RA; ++a) acc[a * (a + 1) + b] = __fma_rn(av[a], yb, acc[a * (a + 1) + b]);
          }
          if (gw == 0) {
            const double sd = sel_sd[r0 + r];
#pragma unroll
            for (int m = 0; m < NV; ++m)
              if (KMAX >= 32 || lane < KMAX) bv[m] = __fma_rn(y[lane + 32 * m], sd, bv[m]);
          }
        }
        gsync();
      }
      nloc += cnt;
    }

    if (nloc == 0) {
      // LETKF.hpp:167-190: no local obs, x' *= sqrt(rho) (RTPS: unchanged).
      const double sr = rtps ? 1.0 : sqrt(prm.rho);
      for (int e = t; e < prm.n_var * k; e += 32 * NW) {
        const int v = e / k, i = e - v * k;
        const int64_t s = base + (int64_t)v * prm.var_stride;
        mg::letkf_store(prm, s * k + i, prm.xmean[s] + Xp[s * k + i] * sr);
      }
      if (t == 0) atomicAdd(prm.n_empty, 1ull);
      gsync();
      continue;
    }
#pragma unroll
    for (int a = 0; a < RA; ++a)
#pragma unroll
      for (int b = 0; b < 2 * (a + 1); ++b)
        if (TI * a + li == TJ * b + lj) acc[a * (a + 1) + b] += diag;

    // ---- A = U D U^T, columns k-1 .. 0; b <- U^-1 b on the way ----
    bool ok = true;
#pragma unroll
    for (int ab = RA - 1; ab >= 0; --ab) {
      for (int jj = TI - 1; jj >= 0; --jj) {
        const int j = ab * TI + jj;
        if (j >= k) continue;
        double* rw = row + (jj & 1) * KMAX;
        if (li == jj) {
#pragma unroll
          for (int b = 0; b < 2 * (ab + 1); ++b) rw[TJ * b + lj] = acc[ab * (ab + 1) + b];
        }
        gsync();
        double d = rw[j];
        if (!mg::pivot_ok(d)) {
          ok = false;
          d = 1.0;
        }
        if (gw == 0) {
          const double r = mg::recip_fp64(d);
          // u of column j: computed by the first warp, read by the group
          const double zj = __shfl_sync(0xffffffffu, bv[(ab * TI) / 32], j & 31);
#pragma unroll
          for (int m = 0; m < NV; ++m) {
            const int l = lane + 32 * m;
            if (l < j) {
              const double u = rw[l] * r;
              S[j * LDS + l] = u;
              bv[m] = __fma_rn(-u, zj, bv[m]);
            }
          }
          if (lane == 0) {
            dinv[j] = r;
            dval[j] = d;
          }
        }
        gsync();
        if (j > 0) {
          double ui[RA];
#pragma unroll
          for (int a = 0; a <= ab; ++a) ui[a] = S[j * LDS + TI * a + li];
#pragma unroll
          for (int b = 0; b < 2 * (ab + 1); ++b) {
            const double rb = rw[TJ * b + lj];
#pragma unroll
            for (int a = b / 2; a <= ab; ++a) acc[a * (a + 1) + b] = __fma_rn(-ui[a], rb, acc[a * (a + 1) + b]);
          }
        }
      }
    }
    if (!ok && t == 0) atomicExch(prm.status, 1);
    gsync();

    // ---- wa = U^-T D^-1 z (first warp) and M's row sums (last warp) ----
    if (NW == 1 || gw == 0 || (gw == NW - 1 && upd_compat)) {
      const bool do_wa = gw == 0, do_rs = gw == NW - 1 && upd_compat;
      double x[NV], y[NV];
#pragma unroll
      for (int m = 0; m < NV; ++m) {
        const int i = lane + 32 * m;
        x[m] = (do_wa && i < k) ? bv[m] * dinv[i] : 0.0;
        y[m] = (do_rs && i < k) ? rsqrt(dval[i]) : 0.0;
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
              const double s = S[i * LDS + l];
              if (do_wa) x[q] = __fma_rn(-s, xl, x[q]);
              if (do_rs) y[q] = __fma_rn(-s, yl, y[q]);
            }
          }
        }
      }
#pragma unroll
      for (int m = 0; m < NV; ++m) {
        const int i = lane + 32 * m;
        if (i < k) {
          if (do_wa) wa_s[i] = sc * x[m];
          if (do_rs) rs_s[i] = cw * y[m];
        }
      }
    }
    gsync();

    // ---- update ----
    if (upd_compat) {  // xa_i = (xm + x'_i wa_i) + x'_i sum_j W_ij, LETKF.hpp:232-238
      for (int e = t; e < prm.n_var * k; e += 32 * NW) {
        const int v = e / k, i = e - v * k;
        const int64_t s = base + (int64_t)v * prm.var_stride;
        const double xp = Xp[s * k + i];
        mg::letkf_store(prm, s * k + i, (prm.xmean[s] + xp * wa_s[i]) + xp * rs_s[i]);
      }
    } else {  // xa = xm + x' wa + W^T x', one warp per variable
      for (int v = gw; v < prm.n_var; v += NW) {
        const int64_t s = base + (int64_t)v * prm.var_stride;
        double x[NV], inc = 0.0, sb = 0.0, sa = 0.0;
#pragma unroll
        for (int m = 0; m < NV; ++m) {
          const int i = lane + 32 * m;
          x[m] = i < k ? Xp[s * k + i] : 0.0;
          if (i < k) inc = __fma_rn(x[m], wa_s[i], inc);
          sb = __fma_rn(x[m], x[m], sb);
        }
#pragma unroll
        for (int m = NV - 1; m >= 0; --m) {  // U^-1 x
          for (int jl = 31; jl >= 0; --jl) {
            const int j = 32 * m + jl;
            if (j >= k || j == 0) continue;
            const double xj = __shfl_sync(0xffffffffu, x[m], jl);
#pragma unroll
            for (int q = 0; q <= m; ++q) {
              const int l = lane + 32 * q;
              if (l < j) x[q] = __fma_rn(-S[j * LDS + l], xj, x[q]);
            }
          }
        }
#pragma unroll
        for (int m = 0; m < NV; ++m) {
          const int i = lane + 32 * m;
          x[m] = i < k ? cw * x[m] * rsqrt(dval[i]) : 0.0;
          sa = __fma_rn(x[m], x[m], sa);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          inc += __shfl_xor_sync(0xffffffffu, inc, off);
          sb += __shfl_xor_sync(0xffffffffu, sb, off);
          sa += __shfl_xor_sync(0xffffffffu, sa, off);
        }
        double f = 0.0;  // relaxation to prior spread: factor - 1
        if (rtps) {
          sb = sqrt(sb / (k - 1));
          sa = sqrt(sa / (k - 1));
          f = (sa > 0.0) ? prm.rho * (sb - sa) / sa : 0.0;
        }
        const double xm = prm.xmean[s];
#pragma unroll
        for (int m = 0; m < NV; ++m) {
          const int i = lane + 32 * m;
          if (i < k) mg::letkf_store(prm, s * k + i, ((xm + inc) + x[m]) + f * x[m]);
        }
      }
    }
    if (t == 0) {
      atomicAdd(prm.total_local, (unsigned long long)nloc);
      atomicMax(prm.max_local, nloc);
    }
    gsync();
  }
}

template <int KMAX, int NW>
cudaError_t launch(const LetkfParams& prm, int num_sms, cudaStream_t s) {
  const size_t smem = Cfg<KMAX, NW>::BYTES;
  cudaError_t e = cudaFuncSetAttribute(letkf_chol_kernel<KMAX, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, letkf_chol_kernel<KMAX, NW>, kThreads, smem);
  if (e != cudaSuccess) return e;
  const int64_t want = (prm.npoints + Cfg<KMAX, NW>::GROUPS - 1) / Cfg<KMAX, NW>::GROUPS;
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>((int64_t)std::max(per_sm, 1) * num_sms, want));
  letkf_chol_kernel<KMAX, NW><<<(unsigned)grid, kThreads, smem, s>>>(prm);
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

}  // namespace

namespace mg {

cudaError_t letkf_chol_launch(const LetkfParams& prm, int num_sms, cudaStream_t s) {
  // Up to two points per SM, four warps an analysis: with one, a point has a
  // single scheduler and the others idle (304 points, k = 20, 3000 local obs:
  // 2901 us by one warp, 1552 by four; 28 local obs 53 and 36).  From three per
  // SM the idle lanes of the wider grid cost more than they bring where the
  // lists are short (456 points, k = 9, 4 local obs: 15.8 and 17.9 us; 608 points,
  // 28 local obs: 26 and 28), and more points always favour one warp (5000 points,
  // k = 32, 28 local obs: 337 and 458 us).
  const bool few = prm.npoints <= 2 * num_sms;
  if (prm.k <= 16) return few ? launch<16, 4>(prm, num_sms, s) : launch<16, 1>(prm, num_sms, s);
  if (prm.k <= 32) return few ? launch<32, 4>(prm, num_sms, s) : launch<32, 1>(prm, num_sms, s);
  if (prm.k <= 64) return launch<64, 4>(prm, num_sms, s);
  return launch<96, 4>(prm, num_sms, s);
}

}  // namespace mg
