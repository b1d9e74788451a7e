// Local observation search (LETKF.hpp:159-165 with Location::distance_to).
//
// Grid coordinates: exact integer distances, a CTA per 8 x 8 points, obs
// scanned in order and compacted with warp ballots so every list comes out
// in obs order, as the reference builds it.
//
// Geographic coordinates: a device-built spatial hash of 1 x 1 degree cells.
// Each query column visits only the cells its radius can reach (latitude
// band bound plus a longitude bound from the haversine inequality
// a >= cos(lat_c) cos(lat_o) sin^2(dlon/2)); the reachable cells of one
// latitude band are one or two contiguous runs of the cell-sorted obs, which
// the whole CTA sweeps as one sequence.  The test on a candidate is the squared
// half chord |u_c - u_o|^2 / 4 between unit vectors (u_o stored with the hash),
// compared with the radius's: haversine <= r  <=>  half chord^2 <=
// sin^2(r/2R), with an absolute error near 1e-16 against a band of 2e-9
// relative in chord^2 (radii of 50 km or more; smaller radii evaluate the
// reference haversine instead).  Lists are sorted by obs index.
// Pairs within 1e-9 relative of the radius are re-decided on the host with
// the reference expression (glibc libm), so the selection is bit-exact
// whatever the device's transcendental rounding.
//
// What bounds it is the FP64 pipe (an instruction of a warp holds its
// scheduler for 64 cycles), so FP64 is kept for what needs it: the windows of
// all columns come from one kernel that fills its lanes (made by one warp of
// each column's CTA, twice, they were half of the search), a candidate is
// tested in FP32 and in FP64 only within FP32's error of the radius, and the
// distance takes about 24 instructions.  64800 columns, 500k obs, 50M list
// entries: count 3.06 -> 0.37 ms, fill 5.91 -> 2.76 ms, windows 0.12 ms.
#include <algorithm>
#include <cmath>
#include <vector>

#include "mg_internal.h"

namespace {

constexpr double kPi = 3.14159265358979323846;
constexpr double kEarthKm = 6371.0;
constexpr int kNBand = 180, kNLonCell = 360, kNCell = kNBand * kNLonCell;
constexpr int kMaxList = 32768;   // longest per-column list sorted in shared memory (128 KB)
constexpr int kBorderCap = 65536; // near-threshold pairs re-decided on the host
constexpr double kBorderRel = 1e-9;

struct BorderRec {
  int64_t col;
  int64_t obs;
  double clat, clon, olat, olon;
};

// ---------------------------------------------------------------- grid ----
__global__ void select_grid_kernel(int nx, int ny, const int32_t* __restrict__ obs_xy, int64_t p,
                                   double radius, const int64_t* __restrict__ offsets,
                                   int64_t* __restrict__ counts, int32_t* __restrict__ idx) {
  const int lane = threadIdx.x & 31;
  const int64_t npt = (int64_t)nx * ny;
  const int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (g >= npt) return;
  const int gx = (int)(g % nx), gy = (int)(g / nx);
  int64_t w = offsets ? offsets[g] : 0;
  for (int64_t o0 = 0; o0 < p; o0 += 32) {
    const int64_t o = o0 + lane;
    bool in = false;
    if (o < p) {
      const double dx = (double)(gx - obs_xy[2 * o]);
      const double dy = (double)(gy - obs_xy[2 * o + 1]);
      in = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy))) <= radius;
    }
    const unsigned b = __ballot_sync(0xffffffffu, in);
    if (idx && in) idx[w + __popc(b & ((1u << lane) - 1u))] = (int32_t)o;
    w += __popc(b);
  }
  if (!offsets && lane == 0) counts[g] = w;
}

// The same lists for 0 <= radius < 2^26 without FP64 (two lanes per clock per
// SM) and without testing every obs at every point: the squared distance is
// an integer below 2^53, exact in the reference's double arithmetic, and
// sqrt is monotone, so sqrt(m) <= radius is m <= r2, r2 the largest integer
// whose rounded square root is within the radius.  One CTA owns 8 x 8
// points: the obs inside its box widened by the radius are compacted in obs
// order (slabs of 256), then each warp tests that short list for the 8
// points of one row.  (144 x 72 points, 2592 obs, radius 6: 12 us a pass, 734 us
// over all pairs.)
constexpr int kSelTile = 8, kSelCap = 1024;
__global__ void __launch_bounds__(256) select_grid_tile_kernel(int nx, int ny, const int32_t* __restrict__ obs_xy,
                                                               int64_t p, int64_t ri, int64_t r2,
                                                               const int64_t* __restrict__ offsets,
                                                               int64_t* __restrict__ counts,
                                                               int32_t* __restrict__ idx) {
  __shared__ int cx[kSelCap], cy[kSelCap], co[kSelCap];
  __shared__ int wcnt[2][8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = blockIdx.x * kSelTile, y0 = blockIdx.y * kSelTile;
  const int gy = y0 + warp;
  int64_t w[kSelTile];
#pragma unroll
  for (int q = 0; q < kSelTile; ++q)
    w[q] = (offsets && x0 + q < nx && gy < ny) ? offsets[(int64_t)gy * nx + x0 + q] : 0;
  int n = 0, ph = 0;
  for (int64_t o0 = 0; o0 < p; o0 += 256, ph ^= 1) {
    const int64_t o = o0 + tid;
    int x = 0, y = 0;
    bool in = false;
    if (o < p) {
      x = obs_xy[2 * o];
      y = obs_xy[2 * o + 1];
      in = x >= x0 - ri && x <= x0 + kSelTile - 1 + ri && y >= y0 - ri && y <= y0 + kSelTile - 1 + ri;
    }
    const unsigned b = __ballot_sync(0xffffffffu, in);
    if (lane == 0) wcnt[ph][warp] = __popc(b);
    __syncthreads();
    int pos = n + __popc(b & ((1u << lane) - 1u));
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (q < warp) pos += wcnt[ph][q];
      n += wcnt[ph][q];
    }
    if (in) {
      cx[pos] = x;
      cy[pos] = y;
      co[pos] = (int)o;
    }
    if (n <= kSelCap - 256 && o0 + 256 < p) continue;
    __syncthreads();
    if (gy < ny) {
      for (int c0 = 0; c0 < n; c0 += 32) {
        const int c = c0 + lane;
        int64_t dx0 = 0, d2y = INT64_MAX;
        int ob = 0;
        if (c < n) {
          dx0 = (int64_t)x0 - cx[c];
          const int64_t dy = (int64_t)gy - cy[c];
          d2y = dy * dy;
          ob = co[c];
        }
#pragma unroll
        for (int q = 0; q < kSelTile; ++q) {
          const int64_t dx = dx0 + q;
          const bool hit = d2y <= r2 && dx * dx <= r2 - d2y && x0 + q < nx;
          const unsigned m = __ballot_sync(0xffffffffu, hit);
          if (idx && hit) idx[w[q] + __popc(m & ((1u << lane) - 1u))] = ob;
          w[q] += __popc(m);
        }
      }
    }
    n = 0;
    __syncthreads();
  }
  if (!offsets && lane == 0 && gy < ny) {
#pragma unroll
    for (int q = 0; q < kSelTile; ++q)
      if (x0 + q < nx) counts[(int64_t)gy * nx + x0 + q] = w[q];
  }
}

cudaError_t launch_select_grid(int nx, int ny, const int32_t* obs_xy, int64_t p, double radius,
                               const int64_t* offsets, int64_t* counts, int32_t* idx, cudaStream_t s) {
  const int64_t ty = (ny + kSelTile - 1) / kSelTile;
  if (radius >= 0.0 && radius < (double)(1 << 26) && ty <= 65535) {
    int64_t r2 = (int64_t)(radius * radius) + 4;
    while (std::sqrt((double)r2) > radius) --r2;
    const dim3 grid((nx + kSelTile - 1) / kSelTile, (unsigned)ty);
    select_grid_tile_kernel<<<grid, 256, 0, s>>>(nx, ny, obs_xy, p, (int64_t)radius, r2, offsets, counts, idx);
  } else {
    const unsigned blocks = (unsigned)(((int64_t)nx * ny + 7) / 8);
    select_grid_kernel<<<blocks, 256, 0, s>>>(nx, ny, obs_xy, p, radius, offsets, counts, idx);
  }
  MG_COUNT_LAUNCH();
  return cudaGetLastError();
}

// ----------------------------------------------------------- geographic ---
__device__ __forceinline__ int cell_of(double lat, double lon) {
  int band = (int)floor(lat + 90.0);
  band = band < 0 ? 0 : (band >= kNBand ? kNBand - 1 : band);
  double l = lon - 360.0 * floor(lon / 360.0);
  int c = (int)floor(l);
  c = c < 0 ? 0 : (c >= kNLonCell ? kNLonCell - 1 : c);
  return band * kNLonCell + c;
}

// Location::haversine (Location.hpp:349-357) with the device's libm.
__device__ __forceinline__ double haversine_dev(double lat1, double lon1, double lat2, double lon2) {
  const double dlat = (lat2 - lat1) * kPi / 180.0;
  const double dlon = (lon2 - lon1) * kPi / 180.0;
  const double s1 = sin(dlat / 2), s2 = sin(dlon / 2);
  const double a = s1 * s1 + cos(lat1 * kPi / 180.0) * cos(lat2 * kPi / 180.0) * s2 * s2;
  return kEarthKm * (2 * atan2(sqrt(a), sqrt(1 - a)));
}

__global__ void cell_count_kernel(const double* __restrict__ lat, const double* __restrict__ lon,
                                  int64_t p, unsigned long long* __restrict__ cnt) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < p; o += stride)
    atomicAdd(&cnt[cell_of(lat[o], lon[o])], 1ull);
}

__device__ __forceinline__ double3 unit_vec(double lat, double lon) {
  double sa, ca, so, co;
  sincos(lat * kPi / 180.0, &sa, &ca);
  sincos(lon * kPi / 180.0, &so, &co);
  return make_double3(ca * co, ca * so, sa);
}

// Cell-sorted obs (half unit vector in FP32, obs index in w) and, in obs
// order, the half unit vectors in FP64 (w unused: one 32-byte sector each).
// Halved, the vectors' squared distance is the squared half chord.
struct CellObs {
  float4* cell;
  double2* half;  // two per obs
};

// Obs into their cells (positions from the cell starts), by the first `blocks` CTAs.
__device__ __forceinline__ void cell_scatter(const double* __restrict__ lat, const double* __restrict__ lon,
                                             int64_t p, const int64_t* __restrict__ start,
                                             unsigned long long* __restrict__ cursor, const CellObs& co, int blocks) {
  const int64_t stride = (int64_t)blocks * blockDim.x;
  for (int64_t o = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; o < p; o += stride) {
    const int c = cell_of(lat[o], lon[o]);
    const int64_t pos = start[c] + (int64_t)atomicAdd(&cursor[c], 1ull);
    const double3 u = unit_vec(lat[o], lon[o]);
    const double hx = 0.5 * u.x, hy = 0.5 * u.y, hz = 0.5 * u.z;
    co.cell[pos] = make_float4((float)hx, (float)hy, (float)hz, __int_as_float((int)o));
    co.half[2 * o] = make_double2(hx, hy);
    co.half[2 * o + 1] = make_double2(hz, 0.0);
  }
}

// What one search fixes for all columns.
struct GeoRule {
  double theta_deg, a_r;   // the radius as an angle, sin^2 of half of it
  double rlo, rhi;         // the radius less and plus the border
  double h2lo, h2hi;       // their squared half chords
  float f_in, f_out;       // FP32: surely inside up to, surely outside above
  int chord;               // the chord test decides (else the haversine)
  int nslot;               // latitude bands a column can reach, at most
  double cosb[91];         // cos of whole degrees
};

GeoRule geo_rule(double radius_km) {
  GeoRule g;
  const double theta = radius_km / kEarthKm;
  g.theta_deg = theta * 180.0 / kPi;
  const double sh = std::sin(0.5 * theta);
  g.a_r = sh * sh;
  g.rlo = radius_km * (1.0 - kBorderRel);
  g.rhi = radius_km * (1.0 + kBorderRel);
  const double slo = std::sin(0.5 * g.rlo / kEarthKm), shi = std::sin(0.5 * g.rhi / kEarthKm);
  g.h2lo = slo * slo;
  g.h2hi = shi * shi;
  g.chord = radius_km >= 50.0;
  // FP32 half chords: each coordinate (at most 1/2) is off by at most 2^-26,
  // so a difference vector by at most sqrt(3) 2^-25 = 5.2e-8, and the
  // subtraction, the squares and their sum add at most 4e-7 relative in the
  // square; 1e-7 and 1e-6 cover both.
  const double d = 1e-7, in = slo > d ? (slo - d) * (slo - d) * (1.0 - 1e-6) : -1.0;
  g.f_in = g.chord ? (float)in : -1.0f;
  g.f_out = (float)((shi + d) * (shi + d) * (1.0 + 1e-6));
  g.nslot = std::min(kNBand, (int)std::floor(2.0 * g.theta_deg + 2e-6) + 2);
  for (int e = 0; e <= 90; ++e) g.cosb[e] = std::cos(e * kPi / 180.0);
  return g;
}

// Search plans: per column the half unit vector, the first reachable latitude
// band, and per band the longitude window as its first and last cell (first >
// last: it wraps; kNoWindow: none).
struct GeoPlan {
  double* hx;
  double* hy;
  double* hz;
  int32_t* b0;
  uint32_t* win;  // nslot per column
};
constexpr uint32_t kNoWindow = 0xffffffffu;

// The scatter and, by the CTAs after its own, the columns' plans (in a launch
// of their own a small search took one launch more than it has to): four
// threads per column, each every fourth band.
__global__ void __launch_bounds__(256) scatter_plan_kernel(const double* __restrict__ obs_lat,
                                                           const double* __restrict__ obs_lon, int64_t p,
                                                           const int64_t* __restrict__ start,
                                                           unsigned long long* __restrict__ cursor, CellObs co,
                                                           int scatter_blocks, const double* __restrict__ col_lat,
                                                           const double* __restrict__ col_lon, int64_t ncol,
                                                           const __grid_constant__ GeoRule g, GeoPlan pl) {
  if ((int)blockIdx.x < scatter_blocks) {
    cell_scatter(obs_lat, obs_lon, p, start, cursor, co, scatter_blocks);
    return;
  }
  const int64_t t = (int64_t)((int)blockIdx.x - scatter_blocks) * blockDim.x + threadIdx.x;
  const int64_t col = t >> 2;
  const int q = (int)(t & 3);
  if (col >= ncol) return;
  const double la = col_lat[col], lo = col_lon[col];
  int b0 = (int)floor(la + 90.0 - g.theta_deg - 1e-6);
  int b1 = (int)floor(la + 90.0 + g.theta_deg + 1e-6);
  b0 = b0 < 0 ? 0 : b0;
  b1 = b1 >= kNBand ? kNBand - 1 : b1;
  double sa, cosc;
  sincos(la * kPi / 180.0, &sa, &cosc);
  if (q == 0) {
    double so, cl;
    sincos(lo * kPi / 180.0, &so, &cl);
    pl.hx[col] = 0.5 * (cosc * cl);
    pl.hy[col] = 0.5 * (cosc * so);
    pl.hz[col] = 0.5 * sa;
    pl.b0[col] = b0;
  }
  for (int i = q; i < g.nslot; i += 4) {
    const int band = b0 + i;
    uint32_t w = kNoWindow;
    if (band <= b1) {
      const int e0 = band - 90, em = e0 >= 0 ? e0 + 1 : -e0;  // the band's larger |latitude|
      const double denom = cosc * g.cosb[em];
      int c0 = 0, c1 = kNLonCell - 1;
      if (denom > g.a_r * (1.0 + 1e-6)) {
        const double sarg = sqrt(g.a_r / denom) * (1.0 + 1e-9);
        if (sarg < 1.0) {
          const double dl = 2.0 * asin(sarg) * 180.0 / kPi + 1e-6;
          if (2.0 * dl + 2.0 < 360.0) {
            c0 = (int)floor(lo - dl);
            c1 = (int)floor(lo + dl);
          }
        }
      }
      // The cells c0..c1 (mod 360) as at most two contiguous runs of obs.
      if (c1 - c0 + 1 >= kNLonCell) {
        w = (uint32_t)(kNLonCell - 1) << 16;
      } else {
        const int a0 = ((c0 % kNLonCell) + kNLonCell) % kNLonCell;
        const int a1 = ((c1 % kNLonCell) + kNLonCell) % kNLonCell;
        w = (uint32_t)a0 | ((uint32_t)a1 << 16);
      }
    }
    pl.win[col * g.nslot + i] = w;
  }
}

constexpr int kMaxRuns = 2 * kNBand;

// One column's plan in shared memory: its candidates as one sequence of the
// runs, pre[r] of them before run r.
struct ColPlan {
  double la, lo, hx, hy, hz;
  float fx, fy, fz;
  int nrun;
  int64_t first[kMaxRuns];
  int32_t pre[kMaxRuns + 1];
};

// By warp 0.
__device__ void load_plan(int64_t col, double la, double lo, const GeoRule& g, const GeoPlan& gp,
                          const int64_t* __restrict__ start, ColPlan& pl) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    pl.la = la;
    pl.lo = lo;
    pl.hx = gp.hx[col];
    pl.hy = gp.hy[col];
    pl.hz = gp.hz[col];
    pl.fx = (float)pl.hx;
    pl.fy = (float)pl.hy;
    pl.fz = (float)pl.hz;
    pl.nrun = 2 * g.nslot;
    pl.pre[0] = 0;
  }
  const int b0 = gp.b0[col];
  int total = 0;
  for (int s0 = 0; s0 < g.nslot; s0 += 32) {
    const int s = s0 + lane;
    int64_t f0 = 0, f1 = 0;
    int n0 = 0, n1 = 0;
    const uint32_t w = s < g.nslot ? gp.win[col * g.nslot + s] : kNoWindow;
    if (w != kNoWindow) {
      const int bb = (b0 + s) * kNLonCell, a0 = (int)(w & 0xffffu), a1 = (int)(w >> 16);
      f0 = start[bb + a0];
      if (a0 <= a1) {
        n0 = (int)(start[bb + a1 + 1] - f0);
      } else {
        n0 = (int)(start[bb + kNLonCell] - f0);
        f1 = start[bb];
        n1 = (int)(start[bb + a1 + 1] - f1);
      }
    }
    int inc = n0 + n1;  // inclusive scan over the lanes
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, d);
      if (lane >= d) inc += v;
    }
    if (s < g.nslot) {
      pl.first[2 * s] = f0;
      pl.first[2 * s + 1] = f1;
      pl.pre[2 * s + 1] = total + inc - n1;
      pl.pre[2 * s + 2] = total + inc;
    }
    total += __shfl_sync(0xffffffffu, inc, 31);
  }
}

// The FP64 test of a candidate within FP32's error of the radius, and of every
// candidate near a small radius (out of line: a predicated FP64 instruction
// would hold the pipe for every candidate).  +1 inside, 0 within 1e-9 relative
// of the radius, -1 outside.
__device__ __noinline__ int test_fp64(const ColPlan& pl, const GeoRule& g, const CellObs& co,
                                      const double* __restrict__ obs_lat, const double* __restrict__ obs_lon, int o) {
  if (g.chord) {
    const double2 xy = co.half[2 * (int64_t)o], zw = co.half[2 * (int64_t)o + 1];
    const double dx = xy.x - pl.hx, dy = xy.y - pl.hy, dz = zw.x - pl.hz;
    const double h2 = dx * dx + dy * dy + dz * dz;
    return h2 <= g.h2lo ? 1 : (h2 <= g.h2hi ? 0 : -1);
  }
  const double d = haversine_dev(pl.la, pl.lo, obs_lat[o], obs_lon[o]);
  return d <= g.rlo ? 1 : (d <= g.rhi ? 0 : -1);
}

// Visits every candidate obs of a planned column with the whole CTA and calls
// f(o, cls) with cls = +1 (inside), 0 (border) or -1; every lane of a warp
// takes part in each call (cls = -1 past the end).
template <typename F>
__device__ __forceinline__ void visit_candidates(const ColPlan& pl, const GeoRule& g, const CellObs& co,
                                                 const double* __restrict__ obs_lat,
                                                 const double* __restrict__ obs_lon, F&& f) {
  const int n = pl.pre[pl.nrun];
  const float fx = pl.fx, fy = pl.fy, fz = pl.fz, f_in = g.f_in, f_out = g.f_out;
  int r = 0;
  for (int i0 = threadIdx.x & ~31; i0 < n; i0 += blockDim.x) {
    const int i = i0 + (threadIdx.x & 31);
    int o = -1, cls = -1;
    if (i < n) {
      while (i >= pl.pre[r + 1]) ++r;
      const float4 u = co.cell[pl.first[r] + (i - pl.pre[r])];
      const float dx = u.x - fx, dy = u.y - fy, dz = u.z - fz;
      const float h2 = dx * dx + dy * dy + dz * dz;
      o = __float_as_int(u.w);
      if (h2 <= f_in) cls = 1;
      else if (h2 <= f_out) cls = test_fp64(pl, g, co, obs_lat, obs_lon, o);
    }
    f(o, cls);
  }
}

// 2R asin(h) of a squared half chord h2 <= 1.  Up to h = 0.05 (great-circle
// distances up to about 640 km) asin by its Maclaurin series
// asin h = sum_n (2n)! / (4^n (n!)^2 (2n + 1)) h^(2n+1), through n = 5: the
// first omitted term, 231/13312 h^13, is below 1e-18 of h there; larger h take
// the library asin.  h = sqrt(h2) from an FP32 reciprocal root y by one step
// of third order (h2 y^2 = 1 - e: sqrt(h2) = h2 y (1 + e/2 + 3 e^2/8 + ..), e
// below 2^-21) and one Newton step on the result.
__device__ __forceinline__ double geo_distance(double h2) {
  double h;
  if (h2 > 1e-30) {
    const double y = (double)rsqrtf((float)h2);
    const double t = h2 * y;
    const double e = fma(-t, y, 1.0);
    const double s = fma(t * e, fma(e, 0.375, 0.5), t);
    h = fma(fma(-s, s, h2), 0.5 * y, s);
  } else {
    h = sqrt(h2);
  }
  if (h > 0.05) return 2.0 * kEarthKm * asin(h < 1.0 ? h : 1.0);
  double q = 63.0 / 2816.0;
  q = fma(q, h2, 35.0 / 1152.0);
  q = fma(q, h2, 5.0 / 112.0);
  q = fma(q, h2, 3.0 / 40.0);
  q = fma(q, h2, 1.0 / 6.0);
  return 2.0 * kEarthKm * fma(h * h2, q, h);
}

__device__ __forceinline__ bool key_rejected(const unsigned long long* rej, int nrej,
                                             unsigned long long key) {
  int lo = 0, hi = nrej;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (rej[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo < nrej && rej[lo] == key;
}

__global__ void __launch_bounds__(256) geo_count_kernel(
    const double* __restrict__ col_lat, const double* __restrict__ col_lon, const __grid_constant__ GeoRule g,
    GeoPlan gp, const int64_t* __restrict__ start, CellObs co, const double* __restrict__ obs_lat,
    const double* __restrict__ obs_lon, int64_t* __restrict__ counts, BorderRec* __restrict__ border,
    unsigned long long* __restrict__ nborder) {
  __shared__ int scount;
  __shared__ ColPlan pl;
  const int64_t col = blockIdx.x;
  if (threadIdx.x == 0) scount = 0;
  const double la = col_lat[col], lo = col_lon[col];
  if (threadIdx.x < 32) load_plan(col, la, lo, g, gp, start, pl);
  __syncthreads();
  int mine = 0;
  visit_candidates(pl, g, co, obs_lat, obs_lon, [&](int o, int cls) {
    if (cls >= 0) ++mine;
    if (cls == 0) {
      const unsigned long long slot = atomicAdd(nborder, 1ull);
      if (slot < (unsigned long long)kBorderCap)
        border[slot] = BorderRec{col, (int64_t)o, la, lo, obs_lat[o], obs_lon[o]};
    }
  });
  mine = __reduce_add_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&scount, mine);
  __syncthreads();
  if (threadIdx.x == 0) {
    counts[col] = (int64_t)scount;
    atomicMax(nborder + 1, (unsigned long long)scount);  // the longest list sizes the fill pass's shared memory
  }
}

__global__ void apply_rejections_kernel(const unsigned long long* __restrict__ rej, int nrej,
                                        int64_t* __restrict__ counts) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nrej) atomicAdd(reinterpret_cast<unsigned long long*>(&counts[rej[t] >> 32]),
                          (unsigned long long)-1ll);
}

// Bitonic sort of 256 E keys by the CTA (ascending): thread t holds elements
// E t .. E t + E - 1, so strides below E stay in registers, strides below 32 E
// are shuffles, and only the rest (6 of 55 steps for 1024 keys) go through
// shared memory, `x` with 256 E entries.
template <int E>
__device__ __forceinline__ void sort_keys(int (&v)[E], int32_t* x) {
  const int t = threadIdx.x;
#pragma unroll
  for (int size = 2; size <= 256 * E; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride < E) {
#pragma unroll
        for (int i = 0; i < E; ++i) {
          if (!(i & stride)) {
            const bool up = (((E * t + i) & size) == 0);
            const int a = v[i], b = v[i | stride];
            const int lo = min(a, b), hi = max(a, b);
            v[i] = up ? lo : hi;
            v[i | stride] = up ? hi : lo;
          }
        }
      } else {
        const int d = stride / E;  // the partner's distance in threads
        int w[E];
        if (d < 32) {
#pragma unroll
          for (int i = 0; i < E; ++i) w[i] = __shfl_xor_sync(0xffffffffu, v[i], d);
        } else {
          __syncthreads();
#pragma unroll
          for (int i = 0; i < E; ++i) x[256 * i + t] = v[i];
          __syncthreads();
#pragma unroll
          for (int i = 0; i < E; ++i) w[i] = x[256 * i + (t ^ d)];
        }
        const bool keep_min = (((E * t) & size) == 0) == ((t & d) == 0);
#pragma unroll
        for (int i = 0; i < E; ++i) v[i] = keep_min ? min(v[i], w[i]) : max(v[i], w[i]);
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < E; ++i) x[E * t + i] = v[i];
}

template <int E>
__device__ __noinline__ void sort_list(int32_t* slist, int cnt) {
  int v[E];
#pragma unroll
  for (int i = 0; i < E; ++i) {  // any assignment of the keys to the elements
    const int e = threadIdx.x + 256 * i;
    v[i] = e < cnt ? slist[e] : 0x7fffffff;
  }
  sort_keys<E>(v, slist);
}

__global__ void __launch_bounds__(256) geo_fill_kernel(
    const double* __restrict__ col_lat, const double* __restrict__ col_lon, const __grid_constant__ GeoRule g,
    GeoPlan gp, const int64_t* __restrict__ start, CellObs co, const int64_t* __restrict__ offsets,
    const unsigned long long* __restrict__ rej, int nrej, const double* __restrict__ obs_lat,
    const double* __restrict__ obs_lon, int32_t* __restrict__ idx, double* __restrict__ dist,
    int* __restrict__ overflow, int list_cap) {
  extern __shared__ int32_t slist[];  // list_cap entries, a power of two from 256
  __shared__ int scount;
  __shared__ ColPlan pl;
  const int64_t col = blockIdx.x;
  const int64_t base = offsets[col];
  const int64_t n = offsets[col + 1] - base;
  if (n == 0) return;
  if (n > list_cap) {
    if (threadIdx.x == 0) atomicExch(overflow, 1);
    return;
  }
  if (threadIdx.x == 0) scount = 0;
  const double la = col_lat[col], lo = col_lon[col];
  if (threadIdx.x < 32) load_plan(col, la, lo, g, gp, start, pl);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  visit_candidates(pl, g, co, obs_lat, obs_lon, [&](int o, int cls) {
    bool in = cls >= 0;
    if (cls == 0 && nrej > 0 && key_rejected(rej, nrej, ((unsigned long long)col << 32) | (unsigned)o)) in = false;
    const unsigned m = __ballot_sync(0xffffffffu, in);
    int pos = 0;
    if (lane == 0 && m) pos = atomicAdd(&scount, __popc(m));
    pos = __shfl_sync(0xffffffffu, pos, 0) + __popc(m & ((1u << lane) - 1u));
    if (in && pos < list_cap) slist[pos] = o;
  });
  __syncthreads();
  const int cnt = scount;
  if (cnt != (int)n) {  // count and fill passes disagree: report, write nothing
    if (threadIdx.x == 0) atomicExch(overflow, 2);
    return;
  }
  // Sorted by obs index (obs order, as LETKF.hpp:160-165): in registers up to
  // 2048 entries, else in shared memory.
  if (cnt <= 256) sort_list<1>(slist, cnt);
  else if (cnt <= 512) sort_list<2>(slist, cnt);
  else if (cnt <= 1024) sort_list<4>(slist, cnt);
  else if (cnt <= 2048) sort_list<8>(slist, cnt);
  else {
    int m = 4096;
    while (m < cnt) m <<= 1;
    for (int t = cnt + threadIdx.x; t < m; t += blockDim.x) slist[t] = 0x7fffffff;
    __syncthreads();
    for (int size = 2; size <= m; size <<= 1) {
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int t = threadIdx.x; t < (m >> 1); t += blockDim.x) {
          const int lo_i = 2 * t - (t & (stride - 1));
          const int hi_i = lo_i + stride;
          const bool up = ((lo_i & size) == 0);
          const int a = slist[lo_i], b = slist[hi_i];
          if ((a > b) == up) {
            slist[lo_i] = b;
            slist[hi_i] = a;
          }
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < cnt; t += blockDim.x) {
    const int o = slist[t];
    idx[base + t] = o;
    if (dist) {
      if (g.chord) {  // well conditioned for chords up to the radius
        const double2 xy = co.half[2 * (int64_t)o], zw = co.half[2 * (int64_t)o + 1];
        const double dx = xy.x - pl.hx, dy = xy.y - pl.hy, dz = zw.x - pl.hz;
        dist[base + t] = geo_distance(dx * dx + dy * dy + dz * dz);
      } else {
        dist[base + t] = haversine_dev(la, lo, obs_lat[o], obs_lon[o]);
      }
    }
  }
}

// Host-side reference predicate for near-threshold pairs (Location.hpp:349-357).
double haversine_host(double lat1, double lon1, double lat2, double lon2) {
  auto deg2rad = [](double deg) { return deg * kPi / 180.0; };
  const double dlat = deg2rad(lat2 - lat1);
  const double dlon = deg2rad(lon2 - lon1);
  const double a = std::sin(dlat / 2) * std::sin(dlat / 2) +
                   std::cos(deg2rad(lat1)) * std::cos(deg2rad(lat2)) * std::sin(dlon / 2) *
                       std::sin(dlon / 2);
  const double c = 2 * std::atan2(std::sqrt(a), std::sqrt(1 - a));
  return kEarthKm * c;
}

}  // namespace

namespace mg {

size_t select_grid_bytes(int64_t npt) {
  Carver cv;
  cv.reserve<int64_t>(npt + 1);
  cv.reserve<char>(scan_temp_bytes(npt));
  return cv.off;
}

}  // namespace mg

extern "C" {

int mg_select_grid(mg_context* ctx, int32_t nx, int32_t ny, const int32_t* obs_xy, int64_t p,
                   double radius, int64_t* offsets, int32_t* idx, int64_t cap, int64_t* total) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(nx > 0 && ny > 0 && p >= 0 && offsets && total && (p == 0 || obs_xy),
               "mg_select_grid: bad arguments");
  const int64_t npt = (int64_t)nx * ny;
  const size_t tmpb = mg::scan_temp_bytes(npt);
  void* ws = mg::workspace(ctx, mg::select_grid_bytes(npt));
  if (!ws) return MG_ERR_NOMEM;
  mg::Carver cv{static_cast<char*>(ws), 0};
  int64_t* counts = cv.take<int64_t>(npt + 1);
  void* tmp = cv.take<char>(tmpb);
  MG_TRY_CUDA(cudaMemsetAsync(counts + npt, 0, sizeof(int64_t), ctx->stream));
  MG_TRY_CUDA(launch_select_grid(nx, ny, obs_xy, p, radius, nullptr, counts, nullptr, ctx->stream));
  MG_TRY_CUDA(mg::exclusive_scan(counts, offsets, npt, tmp, tmpb, ctx->stream));
  MG_TRY_CUDA(cudaMemcpyAsync(total, offsets + npt, sizeof(int64_t), cudaMemcpyDeviceToHost,
                              ctx->stream));
  MG_TRY_CUDA(cudaStreamSynchronize(ctx->stream));
  if (*total > cap || (*total > 0 && !idx))
    return mg::fail(ctx, MG_ERR_CAPACITY, "mg_select_grid: index buffer too small");
  if (*total > 0)
    MG_TRY_CUDA(launch_select_grid(nx, ny, obs_xy, p, radius, offsets, nullptr, idx, ctx->stream));
  return MG_OK;
}

int mg_select_geo(mg_context* ctx, const double* col_lat, const double* col_lon, int64_t ncol,
                  const double* obs_lat, const double* obs_lon, int64_t p, double radius_km,
                  int64_t* offsets, int32_t* idx, double* dist_km, int64_t cap, int64_t* total) {
  if (!ctx) return MG_ERR_ARG;
  MG_CHECK_ARG(col_lat && col_lon && ncol > 0 && p >= 0 && offsets && total && radius_km >= 0 &&
                   (p == 0 || (obs_lat && obs_lon)),
               "mg_select_geo: bad arguments");
  MG_CHECK_ARG(radius_km < 0.5 * kPi * kEarthKm, "mg_select_geo: radius must be below a quarter great circle");
  const size_t tmp_cells = mg::scan_temp_bytes(kNCell);
  const size_t tmp_cols = mg::scan_temp_bytes(ncol);
  const size_t tmpb = std::max(tmp_cells, tmp_cols);
  mg::Carver cv;
  cv.reserve<unsigned long long>(kNCell + 1);  // cell counts, then cursor
  cv.reserve<unsigned long long>(kNCell + 1);
  cv.reserve<int64_t>(kNCell + 1);             // cell start
  const GeoRule rule = geo_rule(radius_km);
  cv.reserve<float4>(p + 1);                   // cell-sorted obs
  cv.reserve<double2>(2 * p + 2);              // half unit vectors in obs order
  for (int a = 0; a < 3; ++a) cv.reserve<double>(ncol);  // search plans
  cv.reserve<int32_t>(ncol);
  cv.reserve<uint32_t>((size_t)ncol * rule.nslot);
  cv.reserve<int64_t>(ncol + 1);               // column counts
  cv.reserve<BorderRec>(kBorderCap);
  cv.reserve<unsigned long long>(kBorderCap);  // rejected keys
  cv.reserve<unsigned long long>(2);           // n_border
  cv.reserve<int>(2);                          // overflow flag
  cv.reserve<char>(tmpb);
  void* ws = mg::workspace(ctx, cv.off);
  if (!ws) return MG_ERR_NOMEM;
  cv = mg::Carver{static_cast<char*>(ws), 0};
  auto* ccount = cv.take<unsigned long long>(kNCell + 1);
  auto* ccursor = cv.take<unsigned long long>(kNCell + 1);
  auto* cstart = cv.take<int64_t>(kNCell + 1);
  CellObs co;
  co.cell = cv.take<float4>(p + 1);
  co.half = cv.take<double2>(2 * p + 2);
  GeoPlan plan;
  plan.hx = cv.take<double>(ncol);
  plan.hy = cv.take<double>(ncol);
  plan.hz = cv.take<double>(ncol);
  plan.b0 = cv.take<int32_t>(ncol);
  plan.win = cv.take<uint32_t>((size_t)ncol * rule.nslot);
  auto* counts = cv.take<int64_t>(ncol + 1);
  auto* border = cv.take<BorderRec>(kBorderCap);
  auto* rej = cv.take<unsigned long long>(kBorderCap);
  auto* nborder = cv.take<unsigned long long>(2);
  auto* overflow = cv.take<int>(2);
  void* tmp = cv.take<char>(tmpb);
  cudaStream_t s = ctx->stream;

  // Spatial hash: counting sort of obs into cells.
  MG_TRY_CUDA(cudaMemsetAsync(ccount, 0, sizeof(unsigned long long) * (kNCell + 1), s));
  MG_TRY_CUDA(cudaMemsetAsync(ccursor, 0, sizeof(unsigned long long) * (kNCell + 1), s));
  MG_TRY_CUDA(cudaMemsetAsync(nborder, 0, sizeof(unsigned long long) * 2, s));
  MG_TRY_CUDA(cudaMemsetAsync(overflow, 0, sizeof(int) * 2, s));
  MG_TRY_CUDA(cudaMemsetAsync(counts, 0, sizeof(int64_t) * (ncol + 1), s));
  const unsigned gb = (unsigned)std::min<int64_t>((p + 255) / 256, 152 * 16);
  if (p > 0) {
    cell_count_kernel<<<gb, 256, 0, s>>>(obs_lat, obs_lon, p, ccount);
    MG_COUNT_LAUNCH();
    MG_TRY_CUDA(cudaGetLastError());
    MG_TRY_CUDA(mg::exclusive_scan(reinterpret_cast<const int64_t*>(ccount), cstart, kNCell, tmp,
                                   tmpb, s));
  } else {
    MG_TRY_CUDA(cudaMemsetAsync(cstart, 0, sizeof(int64_t) * (kNCell + 1), s));
  }
  // Pass 1: counts (near-threshold pairs counted and recorded).
  scatter_plan_kernel<<<gb + (unsigned)((4 * ncol + 255) / 256), 256, 0, s>>>(obs_lat, obs_lon, p, cstart, ccursor, co,
                                                                              (int)gb, col_lat, col_lon, ncol, rule,
                                                                              plan);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  geo_count_kernel<<<(unsigned)ncol, 256, 0, s>>>(col_lat, col_lon, rule, plan, cstart, co, obs_lat, obs_lon, counts,
                                                  border, nborder);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  unsigned long long nbm[2] = {0, 0};
  MG_TRY_CUDA(cudaMemcpyAsync(nbm, nborder, sizeof(nbm), cudaMemcpyDeviceToHost, s));
  MG_TRY_CUDA(cudaStreamSynchronize(s));
  const unsigned long long nb = nbm[0], longest = nbm[1];
  if (longest > (unsigned long long)kMaxList)
    return mg::fail(ctx, MG_ERR_CAPACITY, "mg_select_geo: a local list exceeds 32768 obs");
  if (nb > (unsigned long long)kBorderCap)
    return mg::fail(ctx, MG_ERR_CAPACITY, "mg_select_geo: too many near-threshold pairs");
  int nrej = 0;
  if (nb > 0) {
    std::vector<BorderRec> recs(nb);
    MG_TRY_CUDA(cudaMemcpy(recs.data(), border, sizeof(BorderRec) * nb, cudaMemcpyDeviceToHost));
    std::vector<unsigned long long> keys;
    for (const auto& r : recs)
      if (!(haversine_host(r.clat, r.clon, r.olat, r.olon) <= radius_km))
        keys.push_back(((unsigned long long)r.col << 32) | (unsigned long long)(uint32_t)r.obs);
    std::sort(keys.begin(), keys.end());
    nrej = (int)keys.size();
    if (nrej > 0) {
      MG_TRY_CUDA(cudaMemcpy(rej, keys.data(), sizeof(unsigned long long) * nrej,
                             cudaMemcpyHostToDevice));
      apply_rejections_kernel<<<(nrej + 255) / 256, 256, 0, s>>>(rej, nrej, counts);
      MG_COUNT_LAUNCH();
      MG_TRY_CUDA(cudaGetLastError());
    }
  }
  MG_TRY_CUDA(mg::exclusive_scan(counts, offsets, ncol, tmp, tmpb, s));
  MG_TRY_CUDA(cudaMemcpyAsync(total, offsets + ncol, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  MG_TRY_CUDA(cudaStreamSynchronize(s));
  if (*total > cap || (*total > 0 && !idx))
    return mg::fail(ctx, MG_ERR_CAPACITY, "mg_select_geo: index buffer too small");
  if (*total == 0) return MG_OK;
  // Pass 2: fill, sort each list by obs index, distances.
  int smem_entries = 256;
  while ((unsigned long long)smem_entries < longest) smem_entries <<= 1;
  const size_t smem = sizeof(int32_t) * smem_entries;
  MG_TRY_CUDA(cudaFuncSetAttribute(geo_fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
  geo_fill_kernel<<<(unsigned)ncol, 256, smem, s>>>(col_lat, col_lon, rule, plan, cstart, co, offsets, rej, nrej,
                                                    obs_lat, obs_lon, idx, dist_km, overflow, smem_entries);
  MG_COUNT_LAUNCH();
  MG_TRY_CUDA(cudaGetLastError());
  int ovf = 0;
  MG_TRY_CUDA(cudaMemcpyAsync(&ovf, overflow, sizeof(int), cudaMemcpyDeviceToHost, s));
  MG_TRY_CUDA(cudaStreamSynchronize(s));
  if (ovf == 1) return mg::fail(ctx, MG_ERR_CAPACITY, "mg_select_geo: a local list exceeds its sort buffer");
  if (ovf == 2) return mg::fail(ctx, MG_ERR_NUMERIC, "mg_select_geo: count and fill passes disagree");
  return MG_OK;
}

}  // extern "C"
