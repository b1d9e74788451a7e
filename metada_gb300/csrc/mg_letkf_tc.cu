// Batched LETKF local analyses on the tensor cores (mixed precision, Hunt
// transform, k <= 96): the k x k Gram Y'^T R^-1 Y' as tcgen05.mma kind::tf32
// products, the products of the symmetric inverse square root and the update
// X' W as kind::f16 products of FP16 pairs, all with an error-compensated
// 3-pass split (hi*hi + hi*lo + lo*hi, 22 significant bits an operand) and
// accumulated in FP32 in tensor memory.  Replaces the grid loop of
// LETKF::Analyse (LETKF.hpp:101) and the solve and update of updateGridPoint
// (LETKF.hpp:214-238) in the Hunt et al. (2007) form with Gaspari-Cohn
// R-localisation.
//
// What bounds it: one analysis is a chain of about 12 dependent products,
// each a barrier, an MMA burst and a TMEM -> registers -> operand pass, so a
// CTA alone leaves the tensor core and the shared-memory port idle most of
// the time; the time goes down with the analyses resident per SM and with
// the bytes an operand pass moves.  FP16 pairs take half the shared memory
// and half the MMA time of TF32 pairs.  Three instantiations by member slots
// KP, each as many CTAs per SM as its operands and its tensor memory allow:
//  * KP = 64 (k <= 64): 256 threads, 3 CTAs per SM (128 TMEM columns each);
//    Z and Y are stacked as the 128 rows of one operand, so [Z; Y] T is one
//    M = 128 product.
//  * KP = 80 (64 < k <= 80, the high-resolution configuration's k = 80): 384
//    threads, 2 CTAs per SM (256 columns); Z, Y and T are separate operands
//    and [Z; Y] T is two products.
//  * KP = 96 (80 < k <= 96): as KP = 80 with 1 CTA per SM: 96-slot operands
//    and Gram need more than 256 columns.
// The chain is kept short: one CTA barrier per product (a wait that gave up is
// decided on at the next one), the MMAs of a product issued as straight code
// by one thread (as a loop with a lane election each, issuing took 1300
// cycles a product), T stored by rows, the next analysis pulled and the next
// rows of Y' loaded while others are worked on.
// The finish's products are taken transposed, so that each operand is stored
// by rows (16-byte stores), and the mean's increment rides along as a column.
// The Gram's compensated product takes one MMA pass (k <= 64) or two instead
// of three: its third term is the transpose of the second.
// Whole cycles with TF32 pairs (2, 1 and 1 CTAs, k = 80 in 96 slots) -> FP16
// pairs -> the shorter chain -> this finish -> this Gram: 360 x 180 x 10
// points, 4 variables, k = 64, 500k obs, FP32 members: 118.7 -> 91.9 -> 79.8
// -> 73.1 -> 71.5 ms; 360 x 180 x 30 points, k = 80, clustered obs: 819 -> 496
// -> 406 -> 372 -> 370 ms.  Error against 64 bits on a smaller grid: 2.5e-7 ->
// 2.1e-7.
//
// Per local analysis (one CTA, persistent, points pulled in the grid's
// column order from a work counter):
//  1. Gram: the candidate list is filtered and weighted, the kept rows
//     sqrt(w) Y'_o are gathered 32 at a time into a K-major, 128-byte
//     swizzled operand (members x obs) with sqrt(w) d_o as an extra row, and
//     [b | G] = B^T [sqrt(w) d | B] accumulates in TMEM (three rotating
//     buffers; each chunk's rows are loaded while the previous one's MMAs run).
//  2. A = (k-1)/rho I + G.  The ensemble-mean direction 1 is an exact
//     eigenvector of A (Y' 1 = 0, eigenvalue delta) that never reaches the
//     outputs (X' 1 = 0, 1^T b = 0), so the iteration runs on
//     M = P A P / s + 1 1^T / k (P = I - 1 1^T / k), which puts that mode at 1;
//     s = min(||A||_inf, ||PAP||_F) >= lambda_max keeps M's spectrum in (0, 1].
//  3. Coupled Newton-Schulz with scaled steps: T = a I - b Z Y (a, b from
//     ns_coeffs: the classic (3I - Z Y)/2 after scaling Z and Y by sqrt(mu),
//     mu from the known spectrum bounds [delta/s, 1]), [Z; Y] <- [Z; Y] T; it
//     stops once max |Z Y - I| < 0.05 (one more step squares that error).
//     Z -> M^-1/2, and A^-1/2 = (Z - 1 1^T / k) / sqrt(s) on the complement
//     of 1.
//  4. First-order finish from the matrix itself: C = Z^T (P A P) Z, F = C - P
//     (Z and P A P over their powers of s; the wa and W below carry s),
//     W = sqrt((k-1) c) Z (I - F/2), wa = c Z (P - F) Z^T b (c = rho for the
//     reference's inflation placement, else 1).  max |F| is the per-analysis
//     residual.  Analyses whose conditioning bound s / delta is above
//     kMaxCond, whose iteration does not converge or leaves its basin, whose
//     residual is above the gates (kResidMax, kCondResid delta / s) or whose
//     values are not finite are listed and re-run by the SIMT Jacobi kernel.
//  5. Update: D = W^T X'^T (members x variables) on the tensor core, then
//     x_a = x_mean + X' wa + D (+ RTPS relaxation), written in FP64 (or FP32
//     storage).  Points with at most kPre variables take the short finish:
//     E = Z^T [X'^T b] is issued beside the finish's first product,
//     W^T X'^T = cw (E - F^T E / 2) and X' wa = c E^T (I - F) Z^T b, so
//     neither W nor wa is formed.
// Every mbarrier wait is bounded in time; a wait that gives up makes the CTA
// set the status word, drain its own MMAs (bounded) and free its TMEM.
#include <cuda_runtime.h>

#include "mg_internal.h"
#include "mg_letkf.cuh"
#include "mg_f16op.cuh"
#include "mg_tcgen05.cuh"
#include "mg_tf32op.cuh"

namespace {

using namespace mg::t5;

constexpr int kChunk = 32;      // obs per Gram chunk: one 128-byte swizzle atom of TF32
constexpr int kNBuf = 3;        // Gram chunk buffers
constexpr int kSelRing = 512;   // selected-entry ring (a candidate block + carry-over < kChunk)
constexpr int kMaxIt = 14;      // Newton-Schulz iterations before an analysis is handed back
constexpr float kStop = 0.05f;  // max |Z Y - I| that ends the iteration (after one more step)
constexpr float kResidMax = 5e-3f;  // max |F| accepted from the first-order finish
// Accuracy gates.  A is formed in FP32 from the Gram, a backward error of
// about eps32 ||A||, so the symmetric inverse square root carries a relative
// error of about eps32 kappa along the smallest eigenvalues (kappa =
// lambda_max / lambda_min of P A P on the complement of 1); on the GPU,
// analyses with kappa near 300 reached 1.8e-5 against FP64, those below 150
// stayed under 2.2e-6.  The first-order finish adds about 1e-4 (kappa
// max|F|)^2 (CPU model of this kernel's arithmetic).  s / delta >= kappa is
// known before the iteration (s >= lambda_max, lambda_min >= delta), so an
// analysis runs here only when s / delta <= kMaxCond, and its finish is
// accepted only when max|F| <= kCondResid delta / s as well as kResidMax; the
// others go to the SIMT kernel, whose factor rebuild keeps the small
// eigenvalues' relative accuracy.
constexpr float kMaxCond = 100.0f;
constexpr float kCondResid = 0.1f;
// max |Z Y - I| above which the iteration has left its basin (a convergent
// iterate stays below 1); the analysis is handed back at once.
constexpr float kDiverged = 4.0f;
// Powers of two that operands are stored with (mg_f16op.cuh): Z, Y, T, P A P
// and products of theirs stay below about 20 (kMaxCond bounds Z); X' rows are
// taken in units of their variable's largest entry (below 2), so E = Z^T X'^T
// stays below 2^8; F is accepted up to kResidMax.
constexpr float kSc = 64.0f;                  // Z, Y, T, P A P, Q
constexpr float kScX = 32.0f;                 // X', E
constexpr float kScF = 1048576.0f;            // F
constexpr float kUnZ = 1.0f / (kSc * kSc);    // product of two kSc operands
constexpr float kUnE = 1.0f / (kSc * kScX);   // Z^T X'^T
constexpr float kUnD = 1.0f / (kScF * kScX);  // F^T E
constexpr float kUnZF = 1.0f / (kSc * kScF);  // Z F
constexpr int kVarTile = 16;    // variables per update MMA (N): two 8-column TMEM loads
constexpr int kPre = 4;         // variables whose X' rows and means are prefetched during the finish

// Shared and tensor memory of one CTA, by member slots KP.  The operands of
// the solve are K-major FP16 pairs with the 64-byte swizzle (mg_f16op.cuh): a
// slab holds 32 columns of all its rows (64 bytes per row), with a hi and a
// lo copy.
//   KP = 64: STACK (Z in rows 0-63, Y in rows 64-127), T and P A P (64 rows
//   each): 64 KB.  P A P kept as an operand frees the Gram's tensor memory,
//   so the products take its place: 128 columns.
//   KP = 80, 96: Z, Y and T, each KP rows; P A P stays in tensor memory as
//   the Gram: 90 KB and 256 columns, or 108 KB and 512.
// As a 128-row A operand, operands of fewer rows read the bytes that follow;
// those products land in TMEM lanes that nothing reads.
// Gram view of the same region (TF32 with the 128-byte swizzle, whose exponent
// range needs no scale for the obs rows): three chunk buffers, each of 16
// rows (the innovation's hi and lo, 14 unused), the members' hi rows and their
// lo rows, then the selected-entry ring.  B = the first KP + 16 rows, so one
// MMA gives [hi.d_hi, hi.d_lo | hi hi^T] from the hi rows as A and
// [lo.d_hi, . | lo hi^T] from the lo rows; the third term of the compensated
// product, hi lo^T, is the transpose of the second and is added when the Gram
// is read.  KP = 64: hi and lo rows are the two halves of one 128-row A, a
// third of the MMAs that three passes take; else they are two MMAs into two
// column ranges.
template <int KP>
struct Lay {
  static_assert(KP == 64 || KP == 80 || KP == 96, "member slots");
  static constexpr int NG = (KP + 31) / 32;   // 32-column groups = TMEM lane quadrants holding rows
  static constexpr int kThreads = 128 * NG;   // four lane quadrants x NG column groups of warps
  static constexpr int kWarps = kThreads / 32;
  static constexpr bool kStack = KP == 64;    // [Z; Y] as one 128-row operand
  static constexpr int kMinBlocks = kStack ? 3 : (KP == 80 ? 2 : 1);
  static constexpr int kSteps = KP / 16;      // K-steps of a product
  static constexpr uint32_t ZR = kStack ? 128u : (uint32_t)KP;  // rows per slab of Z and Y
  static constexpr uint32_t TR = KP;                            // rows per slab of T (and P A P)
  static constexpr uint32_t kSlabZ = ZR * 64u;
  static constexpr uint32_t kSlabT = TR * 64u;
  static constexpr uint32_t OFF_Z_HI = 0;
  static constexpr uint32_t OFF_Z_LO = NG * kSlabZ;
  static constexpr uint32_t OFF_Y_HI = kStack ? OFF_Z_HI + KP * 64u : 2 * NG * kSlabZ;
  static constexpr uint32_t OFF_Y_LO = kStack ? OFF_Z_LO + KP * 64u : 3 * NG * kSlabZ;
  static constexpr uint32_t OFF_T_HI = (kStack ? 2 : 4) * NG * kSlabZ;
  static constexpr uint32_t OFF_T_LO = OFF_T_HI + NG * kSlabT;
  static constexpr uint32_t OFF_A_HI = OFF_T_LO + NG * kSlabT;  // P A P (KP = 64)
  static constexpr uint32_t OFF_A_LO = OFF_A_HI + NG * kSlabT;
  static constexpr uint32_t kRegion = kStack ? OFF_A_LO + NG * kSlabT : OFF_A_HI;
  static constexpr int kGramRows = 16 + 2 * KP;
  static constexpr int kGramN = KP + 16;      // Gram MMA N: 16 innovation columns, members
  static constexpr uint32_t kGramBuf = kGramRows * 128u;
  static constexpr uint32_t OFF_SEL = kNBuf * kGramBuf;
  static constexpr uint32_t kSelBytes = kSelRing * 12u;  // obs index, sqrt(w), sqrt(w) d
  // Tensor memory: product scratch at column 0 (and a second product at
  // kTmB), the Gram at kTmGram.
  static constexpr uint32_t kTmemCols = kStack ? 128u : (KP == 80 ? 256u : 512u);
  static constexpr uint32_t kTmB = KP == 80 ? 80u : 128u;
  static constexpr uint32_t kTmE = KP;  // E = Z^T X'^T (16 columns) beside the products
  static constexpr uint32_t kTmGram = kStack ? 0u : (KP == 80 ? 160u : 256u);
  static constexpr uint32_t kTmG = kTmGram + 16;  // its member columns
  static constexpr int kLd = KP + 1;              // lo hi^T on its way to be transposed, FP32 in shared memory
  static_assert(KP * kLd * 4 <= kRegion, "transposition buffer");
  static_assert(kGramBuf % 1024 == 0 && kSlabZ % 512 == 0 && kSlabT % 512 == 0, "swizzle atoms are aligned");
  static_assert(OFF_SEL + kSelBytes <= kRegion && (kStack || OFF_SEL + (128 - KP) * 128 <= kRegion),
                "Gram buffers, the ring, and what the last lo rows read as a 128-row A");
  static_assert(kTmGram + kGramN <= kTmemCols && (kStack || kTmB + KP <= kTmGram), "tensor memory");
  static_assert(kSelRing >= kThreads + kChunk, "ring holds a candidate block and the carry-over");
};

// Vectors after the operand region.
template <int KP>
struct Vecs {
  static constexpr int NG = Lay<KP>::NG;
  float b[KP], r[KP], u[KP], v[KP], wa[KP];
  float part[2 * NG][KP];
  float red[32];
  float xsq[kVarTile], inc[kVarTile], fac[kVarTile], one[kVarTile];
  float ssa[NG][kVarTile], sdw[NG][kPre];
  float xu[kVarTile];  // unit of each variable's X' row (slot kPre in the finish: of b)
  double xm[kVarTile];
  double xmpre[kPre];
  float xmh[kPre], xml[kPre];  // xmpre as a sum of two floats
  float xpre[kPre][KP];
  int wcnt[2][Lay<KP>::kWarps];
};

template <int KP>
constexpr size_t smem_bytes() {
  return 1024 + Lay<KP>::kRegion + sizeof(Vecs<KP>);
}
static_assert(3 * (smem_bytes<64>() + 1280) <= 233472 && 2 * (smem_bytes<80>() + 1280) <= 233472,
              "CTAs per SM by shared memory");
static_assert(sizeof(Vecs<80>) >= 48 * 64 && sizeof(Vecs<96>) >= 32 * 64, "the last rows that T reads as a 128-row operand");

// Scaled Newton-Schulz step.  The spectrum of Z Y lies in [l, 1] (l = delta / s
// at the start: P A P >= delta on the complement of 1, s >= lambda_max).  The
// step scales Z and Y by sqrt(mu) before T = (3I - mu Z Y)/2, i.e.
// T = a I - b Z Y with a = 1.5 sqrt(mu), b = 0.5 mu^1.5, where mu equalises
// the map h(e) = e (3 - e)^2 / 4 at both ends of [mu l, mu]:
// mu = 3 (1 - sqrt l) / (1 - l^1.5).  The new interval is [h(mu l), 1].  The
// iteration keeps its fixed point (Z -> M^-1/2) and needs about 4 steps
// instead of 6 at the configurations' conditioning.
__device__ __forceinline__ void ns_coeffs(float& l, float& a, float& b) {
  float mu = 1.0f;
  if (l < 1.0f) {
    const float sl = sqrtf(l);
    mu = fmaxf(3.0f * (1.0f - sl) / (1.0f - l * sl), 1.0f);
  }
  const float smu = sqrtf(mu);
  a = 1.5f * smu;
  b = 0.5f * mu * smu;
  const float ml = fminf(mu * l, 1.0f);
  l = ml * (3.0f - ml) * (3.0f - ml) * 0.25f;
}

// hi + lo + a + b rounded to FP32 from exact partial sums (Knuth's TwoSum): what
// the sum in FP64 gives for FP32 storage, without four instructions of the
// FP64 pipe, each of which holds a scheduler for 64 cycles.
__device__ __forceinline__ float add3(float hi, float lo, float a, float b) {
  const float s1 = __fadd_rn(hi, a), t1 = __fsub_rn(s1, hi);
  const float r1 = __fadd_rn(__fsub_rn(hi, __fsub_rn(s1, t1)), __fsub_rn(a, t1));
  const float s2 = __fadd_rn(s1, b), t2 = __fsub_rn(s2, s1);
  const float r2 = __fadd_rn(__fsub_rn(s1, __fsub_rn(s2, t2)), __fsub_rn(b, t2));
  return __fadd_rn(s2, __fadd_rn(__fadd_rn(r1, r2), lo));
}

// Asynchronous global -> shared copies (no registers held while in flight).
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// FP64 decision for a candidate whose FP32 vertical distance is within 1e-4
// of the support (kept out of line: a predicated FP64 instruction would
// occupy the FP64 pipe for every candidate).
__device__ __noinline__ bool vertical_keep_fp64(int lev, double obs_lev, double vsupport) {
  return fabs((double)lev - obs_lev) <= vsupport;
}

// One analysis of the grid, and where its candidates lie.
struct Item {
  int64_t base, e0, e1;
  int col, lev;  // lev < 0: none left
};

// The next analysis, by one thread: a chain of four dependent global loads.
__device__ __noinline__ void pull(const mg::LetkfParams& prm, Item& it) {
  const unsigned long long n = atomicAdd(prm.next, 1ull);
  if (n >= (unsigned long long)prm.npoints) {
    it.lev = -1;
    return;
  }
  const uint32_t item = (uint32_t)n, nlev = (uint32_t)prm.nlev;  // npoints fits an int32 (redo_out)
  const int lev = (int)(item % nlev);
  const int64_t col = prm.order[item / nlev];
  it.col = (int)col;
  it.lev = lev;
  it.base = prm.col_base[col] + (int64_t)lev * prm.lev_stride;
  int64_t e0 = prm.loc_off[col], e1 = prm.loc_off[col + 1];
  if (prm.lev_boff) {  // only the level buckets that can reach this level
    const int32_t* bo = prm.lev_boff + col * (int64_t)(prm.nlev + 1);
    const double fl = floor((double)lev - prm.vsupport), fh = floor((double)lev + prm.vsupport);
    const int lo = (fl <= 0.0) ? 0 : (int)fl;
    const int hi = (fh >= (double)(prm.nlev - 1)) ? prm.nlev - 1 : (int)fh;
    e1 = e0 + bo[hi + 1];
    e0 = e0 + bo[lo];
  }
  it.e0 = e0;
  it.e1 = e1;
}

template <int KP>
__global__ void __launch_bounds__(Lay<KP>::kThreads, Lay<KP>::kMinBlocks) letkf_tc_kernel(mg::LetkfParams prm) {
  using L = Lay<KP>;
  constexpr int NG = L::NG;
  constexpr int kThreads = L::kThreads;
  constexpr uint32_t ZR = L::ZR, TR = L::TR;
  using h16::get_col8;
  using h16::get_row8;
  using h16::put_col8;
  using h16::put_row8;
  using h16::put_row8x2;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* R = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Vecs<KP>& V = *reinterpret_cast<Vecs<KP>*>(R + L::kRegion);
  unsigned char* const ZH = R + L::OFF_Z_HI;
  unsigned char* const ZL = R + L::OFF_Z_LO;
  unsigned char* const YH = R + L::OFF_Y_HI;
  unsigned char* const YL = R + L::OFF_Y_LO;
  unsigned char* const TH = R + L::OFF_T_HI;
  unsigned char* const TL = R + L::OFF_T_LO;
  unsigned char* const AH = L::kStack ? R + L::OFF_A_HI : YH;
  unsigned char* const AL = L::kStack ? R + L::OFF_A_LO : YL;
  int* const sel_o = reinterpret_cast<int*>(R + L::OFF_SEL);
  float* const sel_sw = reinterpret_cast<float*>(R + L::OFF_SEL + 4 * kSelRing);
  float* const sel_sd = reinterpret_cast<float*>(R + L::OFF_SEL + 8 * kSelRing);
  __shared__ uint64_t mma_bar;
  __shared__ uint64_t buf_bar[kNBuf];
  __shared__ uint32_t tmem_s;
  __shared__ Item s_it;
  __shared__ unsigned s_flag[2];  // of the iteration's parity; the finish uses the first

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform to the compiler
  const int q = warp & 3, g = warp >> 2;  // TMEM lane quadrant, 32-column group
  const int k = prm.k;
  const float ik = 1.0f / (float)k;
  const float* __restrict__ Y = static_cast<const float*>(prm.Y);
  const float* __restrict__ Xp = static_cast<const float*>(prm.Xp);
  const bool r_identity = prm.flags & MG_R_IDENTITY;
  const bool infl_compat = prm.flags & MG_INFL_COMPAT;
  const bool rtps = prm.flags & MG_RTPS;
  const float delta = (infl_compat || rtps) ? (float)(k - 1) : (float)((double)(k - 1) / prm.rho);
  const float sc = infl_compat ? (float)prm.rho : 1.0f;
  const float cw = sqrtf((float)(k - 1) * sc);
  const float hc = (float)(0.5 * prm.hsupport), vc = (float)(0.5 * prm.vsupport), vs = (float)prm.vsupport;
  const bool vec4 = (k & 3) == 0;

  if (tid == 0) {
    mbar_init(&mma_bar, 1);
    for (int b = 0; b < kNBuf; ++b) mbar_init(&buf_bar[b], 1);
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc(&tmem_s, L::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_s;
  const uint32_t tm_row = ((uint32_t)(32 * q) << 16);  // this warp's TMEM lanes
  // Warp-collective TMEM load; a warp that a row guard split (KP = 80) is
  // brought together first.
  auto ld8 = [](uint32_t addr, uint32_t(&v)[8]) {
    if (KP % 32) __syncwarp();
    tmem_ld8(addr, v);
  };
  const uint32_t sR = smem_u32(R);
  const uint32_t sZH = sR + L::OFF_Z_HI, sZL = sR + L::OFF_Z_LO;
  const uint32_t sYH = sR + L::OFF_Y_HI, sYL = sR + L::OFF_Y_LO;
  const uint32_t sTH = sR + L::OFF_T_HI, sTL = sR + L::OFF_T_LO;
  const uint32_t sAH = L::kStack ? sR + L::OFF_A_HI : sYH, sAL = L::kStack ? sR + L::OFF_A_LO : sYL;  // P A P
  constexpr uint32_t kSlabA = L::kStack ? L::kSlabT : L::kSlabZ;
  const uint32_t idescK = h16::idesc_f16_f32(128, KP);
  const uint32_t idescG = idesc_tf32_f32(128, L::kGramN);
  const uint32_t idescU = h16::idesc_f16_f32(128, kVarTile);

  uint32_t mma_ph = 0;      // parity of the next mma_bar phase
  uint32_t gchunk = 0;      // Gram chunks issued by this CTA (buffer rotation)
  bool alive = true;

  const int32_t* __restrict__ lidx = prm.lev_boff ? prm.bidx : prm.loc_idx;
  const double* __restrict__ ldist = prm.lev_boff ? prm.bdist : prm.loc_dist;
  bool pulled = false;  // s_it holds this analysis

  for (;;) {
    cp_async_wait_all();  // a handed-back analysis may leave its prefetch in flight
    if (!pulled) {
      if (tid == 0) pull(prm, s_it);
      __syncthreads();
    }
    pulled = false;
    const int lev = s_it.lev, col = s_it.col;
    if (lev < 0) break;
    const int64_t base = s_it.base, e0 = s_it.e0, e1 = s_it.e1;

    // ---------------- 1. selection and Gram ----------------
    // Rounds: compact candidates into the ring (up to kSelRing - kThreads
    // entries), then emit its chunks; each chunk's rows are loaded into
    // registers while the previous chunk is stored and its MMAs issued.
    int64_t cpos = e0;
    bool ok = true;  // this thread's waits since the last decision
    // A block's indices and distances are loaded one block ahead.
    int o_n = 0;
    double d_n = 0.0;
    auto fetch = [&](int64_t c) {
      if (c + tid < e1) {
        o_n = lidx[c + tid];
        if (ldist) d_n = ldist[c + tid];
      }
    };
    fetch(cpos);
    int nloc = 0, nch = 0, head = 0, nsel = 0, par = 0;
    const int slot = tid & (kChunk - 1), m0 = (tid / kChunk) * 8;  // gather: obs slot x 8 members
    // Raw values: they are scaled when they are stored, so the loads stay in
    // flight until then.
    auto load_rows = [&](int pos, int cnt, float (&x)[8], float& sw, float& sd) {
      if (slot < cnt) {
        const int e = (pos + slot) & (kSelRing - 1);
        const int o = sel_o[e];
        sw = sel_sw[e];
        sd = sel_sd[e];
        const float* yr = Y + (int64_t)o * k;
        if (vec4 && m0 + 8 <= k) {
#pragma unroll
          for (int q4 = 0; q4 < 2; ++q4) {
            const float4 a4 = *reinterpret_cast<const float4*>(yr + m0 + 4 * q4);
            x[4 * q4 + 0] = a4.x; x[4 * q4 + 1] = a4.y; x[4 * q4 + 2] = a4.z; x[4 * q4 + 3] = a4.w;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) x[j] = (m0 + j < k) ? yr[m0 + j] : 0.0f;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = 0.0f;
        sw = 0.0f;
        sd = 0.0f;
      }
    };
    while (alive) {
      while (cpos < e1 && nsel <= kSelRing - kThreads) {
        bool keep = false;
        int o = 0;
        float sw = 0.0f, sd = 0.0f;
        const double d = d_n;
        o = o_n;
        fetch(cpos + kThreads);
        if (cpos + tid < e1) {
          const float4 pk = prm.opack[o];  // (level, 1/sigma^2, innovation, 0) as FP32
          float w = 1.0f;
          keep = true;
          if (prm.obs_lev) {
            const float dl = fabsf((float)lev - pk.x);
            if (dl > vs + 1e-4f) keep = false;
            else if (dl >= vs - 1e-4f) keep = vertical_keep_fp64(lev, prm.obs_lev[o], prm.vsupport);
            if (keep && !r_identity) w *= mg::gaspari_cohn<float>(dl / vc);
          }
          if (keep && !r_identity) {
            if (ldist) w *= mg::gaspari_cohn<float>((float)d / hc);
            w *= pk.y;
            if (!(w > 0.0f)) keep = false;
          }
          if (keep) {
            sw = sqrtf(w);
            sd = sw * pk.z;
          }
        }
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) V.wcnt[par][warp] = __popc(bal);
        __syncthreads();
        int wb = 0, cnt = 0;
#pragma unroll
        for (int w = 0; w < L::kWarps; ++w) {
          if (w < warp) wb += V.wcnt[par][w];
          cnt += V.wcnt[par][w];
        }
        if (keep) {
          const int pos = (head + nsel + wb + __popc(bal & ((1u << lane) - 1u))) & (kSelRing - 1);
          sel_o[pos] = o;
          sel_sw[pos] = sw;
          sel_sd[pos] = sd;
        }
        par ^= 1;  // the counts are read before the next but one block writes its own
        nsel += cnt;
        nloc += cnt;
        cpos += kThreads;
      }
      __syncthreads();  // the ring's entries
      const bool done = cpos >= e1;
      const int nchunks = done ? (nsel + kChunk - 1) / kChunk : nsel / kChunk;
      float x[8], swv, sdv;
      if (nchunks > 0) load_rows(head, nsel < kChunk ? nsel : kChunk, x, swv, sdv);
      for (int c = 0; c < nchunks; ++c) {
        const int b = (int)(gchunk % kNBuf);
        const uint32_t use = gchunk / kNBuf;
        if (use > 0 && !wait_one(&buf_bar[b], (use - 1) & 1u)) ok = false;
        unsigned char* bh = R + b * L::kGramBuf;
        if (m0 < KP) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t off = sw_off(16 + m0 + j, slot, L::kGramRows);
            float h, l;
            split(x[j] * swv, h, l);
            *reinterpret_cast<float*>(bh + off) = h;
            *reinterpret_cast<float*>(bh + off + KP * 128) = l;
          }
        }
        if (m0 == 0) {  // the innovation rows
          float h, l;
          split(sdv, h, l);
          *reinterpret_cast<float*>(bh + sw_off(0, slot, L::kGramRows)) = h;
          *reinterpret_cast<float*>(bh + sw_off(1, slot, L::kGramRows)) = l;
        }
        if (c + 1 < nchunks) {  // next chunk's rows in flight during the barrier and the MMAs
          const int rem = nsel - (c + 1) * kChunk;
          load_rows(head + (c + 1) * kChunk, rem < kChunk ? rem : kChunk, x, swv, sdv);
        }
        if (!operands_ready(ok)) { alive = false; break; }
        if (warp == 0) {
          tc_fence_after();
          const uint32_t a = sR + b * L::kGramBuf;
          if (elect_one()) {
            issue_slab(tmem + L::kTmGram, a + 16 * 128, a, idescG, nch > 0);
            if (!L::kStack) issue_slab(tmem, a + (16 + KP) * 128, a, idescG, nch > 0);
            mma_commit(&buf_bar[b]);
          }
          __syncwarp();
        }
        ++gchunk;
        ++nch;
      }
      if (!alive) break;
      head = (head + nchunks * kChunk) & (kSelRing - 1);
      nsel = (nsel > nchunks * kChunk) ? nsel - nchunks * kChunk : 0;
      if (done) break;
    }
    if (!alive) break;

    if (nloc == 0) {
      // LETKF.hpp:167-190: no local obs, x' *= sqrt(rho) (RTPS: unchanged).
      const double sr = rtps ? 1.0 : sqrt(prm.rho);
      for (int e = tid; e < prm.n_var * k; e += kThreads) {
        const int v = e / k, i = e - v * k;
        const int64_t s = base + (int64_t)v * prm.var_stride;
        mg::letkf_store(prm, s * k + i, prm.xmean[s] + (double)Xp[s * k + i] * sr);
      }
      if (tid == 0) atomicAdd(prm.n_empty, 1ull);
      __syncthreads();
      continue;
    }
    if (warp == 0) {
      if (elect_one()) mma_commit(&mma_bar);
      __syncwarp();
    }
    if (!wait_all(&mma_bar, mma_ph, ok)) { alive = false; break; }
    mma_ph ^= 1u;
    // The next analysis, by a warp that holds no rows in this phase.
    if (tid == kThreads - 1) pull(prm, s_it);
    __syncwarp();  // tensor-memory loads of the whole warp follow
    pulled = true;

    // ---------------- 2. A, b, deflation and scaling ----------------
    // Warps of quadrants 0 .. NG-1 hold rows 0 .. KP-1 (their TMEM lanes),
    // column group g; each walks its 32 columns 8 at a time.
    const bool rowwarp = q < NG;
    const int row = 32 * q + lane;
    const bool rowin = row < KP;  // KP = 80: the last rows of the third quadrant hold nothing
    const int cb = 32 * g, ce = (cb + 32 < KP) ? cb + 32 : KP;
    // lo hi^T -> shared memory, with lo.d_hi as its last column.
    float* const S = reinterpret_cast<float*>(R);
    if (L::kStack ? !rowwarp : rowwarp) {
      const int i = L::kStack ? row - 64 : row;
#pragma unroll 1
      for (int c0 = cb; c0 < ce; c0 += 8) {
        uint32_t v[8];
        ld8(tmem + tm_row + 16 + c0, v);
        tmem_wait_ld();
        if (L::kStack || rowin) {
#pragma unroll
          for (int j = 0; j < 8; ++j) S[i * L::kLd + c0 + j] = __uint_as_float(v[j]);
        }
      }
      if (g == 0) {
        const uint32_t bv = tmem_ld1(tmem + tm_row);
        tmem_wait_ld();
        if (L::kStack || rowin) S[i * L::kLd + KP] = __uint_as_float(bv);
      }
    }
    __syncthreads();
    if (rowwarp) {
      float rs = 0.0f, as = 0.0f, fa = 0.0f;
      const int ri = rowin ? row : 0;
      const float dr = (row < k) ? delta : 0.0f;
#pragma unroll 1
      for (int c0 = cb; c0 < ce; c0 += 8) {
        uint32_t v[8];
        ld8(tmem + tm_row + L::kTmG + c0, v);
        tmem_wait_ld();
        const int dj = row - c0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int c = c0 + j;
          const float gv = __uint_as_float(v[j]) + (S[ri * L::kLd + c] + S[c * L::kLd + ri]);
          v[j] = __float_as_uint(gv);  // zero outside the member block (zero rows)
          const float x = gv + ((dj == j) ? dr : 0.0f);
          rs += x;
          as += fabsf(x);
          fa += x * x;
        }
        if (KP % 32) __syncwarp();
        tmem_st8(tmem + tm_row + L::kTmG + c0, v);
      }
      if (rowin) {
        V.part[g][row] = rs;
        V.part[NG + g][row] = as;
      }
      if (!rowin) fa = 0.0f;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) fa += __shfl_xor_sync(0xffffffffu, fa, off);
      if (lane == 0) V.red[3 * NG + q * NG + g] = fa;  // ||A||_F^2, by warp
      if (g == 0) {
        const uint32_t b0 = tmem_ld1(tmem + tm_row + L::kTmGram), b1 = tmem_ld1(tmem + tm_row + L::kTmGram + 1);
        tmem_wait_ld();
        if (rowin)
          V.b[row] = (row < k) ? __uint_as_float(b0) + (__uint_as_float(b1) + S[row * L::kLd + KP]) : 0.0f;
      }
      tmem_wait_st();
    }
    __syncthreads();
    if (warp < NG) {  // row means r, grand mean c, infinity norm
      const int i = tid;
      float r = 0.0f, ab = 0.0f;
      if (i < k) {
#pragma unroll
        for (int gg = 0; gg < NG; ++gg) {
          r += V.part[gg][i];
          ab += V.part[NG + gg][i];
        }
        r *= ik;
      }
      if (i < KP) V.r[i] = r;
      float sr = r, mx = ab, s2 = r * r;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        sr += __shfl_xor_sync(0xffffffffu, sr, off);
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        s2 += __shfl_xor_sync(0xffffffffu, s2, off);
      }
      if (lane == 0) {
        V.red[warp] = sr;
        V.red[NG + warp] = mx;
        V.red[2 * NG + warp] = s2;
      }
    }
    __syncthreads();
    float cbar = 0.0f, ninf = 0.0f;
#pragma unroll
    for (int gg = 0; gg < NG; ++gg) {
      cbar += V.red[gg];
      ninf = fmaxf(ninf, V.red[NG + gg]);
    }
    cbar *= ik;
    // Row `row` of P A P, columns c0 .. c0+7, from the Gram in TMEM (zero
    // outside the member block).
    auto pap8 = [&](int c0, float (&x)[8]) {
      uint32_t v[8];
      ld8(tmem + tm_row + L::kTmG + c0, v);
      tmem_wait_ld();
      const float ri = rowin ? V.r[row] : 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int c = c0 + j;
        const float av = __uint_as_float(v[j]) + ((c == row) ? delta : 0.0f);
        x[j] = (row < k && c < k) ? (av - ri - V.r[c] + cbar) : 0.0f;
      }
    };
    // Frobenius norm of P A P from the same pass (A symmetric, A 1 = k r):
    // ||P A P||_F^2 = ||A||_F^2 - 2 k sum r_i^2 + k^2 cbar^2.  With A 1 =
    // delta 1 up to rounding the subtracted part is about delta^2, at most
    // 1/k of ||A||_F^2 >= k delta^2, so the difference keeps FP32 accuracy
    // (and s only has to bound lambda_max).
    float fa2 = 0.0f, sr2 = 0.0f;
#pragma unroll
    for (int e = 0; e < NG * NG; ++e) fa2 += V.red[3 * NG + e];
#pragma unroll
    for (int gg = 0; gg < NG; ++gg) sr2 += V.red[2 * NG + gg];
    const float kf = (float)k;
    const float fro = sqrtf(fmaxf(fa2 - 2.0f * kf * sr2 + kf * kf * cbar * cbar, 0.0f));
    const float s = fmaxf(fminf(ninf, fro), 1e-30f);
    const float is = 1.0f / s;
    float lsp = fminf(delta * is, 1.0f);  // lower end of the spectrum of Z Y (upper end 1)
    // Points handed to the SIMT Jacobi kernel: nothing is written for them here.
    auto hand_back = [&]() {
      if (tid == 0) {
        const unsigned long long slot = atomicAdd(prm.n_redo, 1ull);
        prm.redo_out[slot] = (int32_t)(col * prm.nlev + lev);
      }
      __syncthreads();
    };
    const float l0 = lsp;  // delta / s, at most 1 / kappa
    if (!(l0 * kMaxCond >= 1.0f)) {
      hand_back();
      continue;
    }
    float nsa, nsb;
    ns_coeffs(lsp, nsa, nsb);
    // M = PAP / s + 1 1^T / k (identity on unused member slots); Y <- M, T
    // <- T0 = a I - b M, and Z <- T0: the first step's Z (Z = I before it), so
    // that step computes Y T only.  P A P / s is kept for the finish where it
    // has its own operand.  T is symmetric up to rounding and stored as
    // computed (a transposed store took 16 two-byte stores for two of 16
    // bytes; on a CPU model of this arithmetic either gives the same errors).
    if (rowwarp) {
#pragma unroll 1
      for (int c0 = cb; c0 < ce; c0 += 8) {
        float x[8], y[8];
        pap8(c0, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          x[j] *= is * kSc;
          y[j] = (row == c0 + j) ? kSc : 0.0f;
        }
        if (L::kStack && rowin) put_row8(AH, AL, row, c0, TR, x);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int c = c0 + j;
          x[j] = (row < k && c < k) ? x[j] + ik * kSc : y[j];
          y[j] = nsa * y[j] - nsb * x[j];
        }
        if (rowin) {
          put_row8(YH, YL, row, c0, ZR, x);
          put_row8x2(TH, TL, TR, ZH, ZL, ZR, row, c0, y);
        }
      }
    }

    // X' rows and means of the first kPre variables, in flight during the
    // Newton-Schulz iteration (members beyond k read as zero).
    const int npre = (prm.n_var < kPre) ? prm.n_var : kPre;
    for (int e = tid; e < kPre * KP; e += kThreads) {
      const int vv = e / KP, m = e - vv * KP;
      if (vv < npre && m < k) cp_async4(&V.xpre[vv][m], Xp + (base + (int64_t)vv * prm.var_stride) * k + m);
      else V.xpre[vv][m] = 0.0f;
    }
    if (tid < npre) cp_async8(&V.xmpre[tid], prm.xmean + base + (int64_t)tid * prm.var_stride);
    // Points with at most kPre variables take the short finish: E = Z^T X'^T
    // is computed beside Q, and X' W = cw (E - F^T E / 2), so W itself is
    // never formed (one dependent product and two epilogues fewer).
    const bool fast = prm.n_var <= kPre;

    // X' row of variable slot vv (zero beyond k and for unused slots), in
    // units of its largest entry, -> T row vv: one warp.
    auto put_x = [&](int vv, float (&x)[NG]) {
      float mx = 0.0f;
#pragma unroll
      for (int gg = 0; gg < NG; ++gg) mx = fmaxf(mx, fabsf(x[gg]));
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const int ex = min(max((int)(__float_as_uint(mx) >> 23), 6), 253);
      const float inv = kScX * __uint_as_float((uint32_t)(254 - ex) << 23);
#pragma unroll
      for (int gg = 0; gg < NG; ++gg) {
        const int m = lane + 32 * gg;
        uint32_t h, l;
        h16::split2(x[gg] * inv, 0.0f, h, l);
        if (m < KP) {
          const uint32_t o = h16::off(vv, m, TR);
          *reinterpret_cast<uint16_t*>(TH + o) = (uint16_t)h;
          *reinterpret_cast<uint16_t*>(TL + o) = (uint16_t)l;
        }
      }
      if (lane == 0) V.xu[vv] = __uint_as_float((uint32_t)ex << 23);
    };
    // ---------------- 3. coupled Newton-Schulz ----------------
    int its = 0;
    bool stop = false;  // decided from max |Z Y - I| of the current iterate
    bool conv = false;
    bool diverged = false;
    for (;;) {
      // [Z; Y] <- [Z; Y] T (the first step: Y only)
      if (!operands_ready(ok)) { alive = false; break; }
      if (its > 0) {
        const unsigned fl = s_flag[its & 1];
        stop = fl == 0u;
        if (fl & 2u) {
          diverged = true;
          break;
        }
      }
      if (warp == 0) {
        tc_fence_after();
        if (elect_one()) {
          if (stop || its + 1 >= kMaxIt) {  // the last step: Z^T = T^T Z^T, by rows as the finish reads it
            h16::issue3<L::kSteps, L::kSlabT, L::kSlabZ>(tmem, sTH, sTL, sZH, sZL, idescK);
          } else if constexpr (L::kStack) {
            h16::issue3<L::kSteps, L::kSlabZ, L::kSlabT>(tmem, sZH, sZL, sTH, sTL, idescK);
          } else {
            if (its > 0) h16::issue3<L::kSteps, L::kSlabZ, L::kSlabT>(tmem, sZH, sZL, sTH, sTL, idescK);
            h16::issue3<L::kSteps, L::kSlabZ, L::kSlabT>(tmem + L::kTmB, sYH, sYL, sTH, sTL, idescK);
          }
          mma_commit(&mma_bar);
        }
        __syncwarp();
      }
      const bool zstep = its > 0;
      ++its;
      const bool last = stop || its >= kMaxIt;
      conv = stop;
      // This iteration's flags (the last ones were read before the barrier
      // that follows).
      if (tid == 0) s_flag[its & 1] = 0u;
      if (!wait_one(&mma_bar, mma_ph)) ok = false;
      mma_ph ^= 1u;
      if (!last) {
        if (L::kStack && (zstep || !rowwarp)) {  // all warps: rows 0-63 Z, 64-127 Y
#pragma unroll 1
          for (int c0 = cb; c0 < ce; c0 += 8) {
            uint32_t v[8];
            ld8(tmem + tm_row + c0, v);
            tmem_wait_ld();
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(v[j]) * (kUnZ * kSc);
            put_row8(ZH, ZL, 32 * q + lane, c0, ZR, x);
          }
        } else if (!L::kStack && rowwarp) {  // Z from the first product, Y from the second
#pragma unroll 1
          for (int c0 = cb; c0 < ce; c0 += 8) {
            uint32_t v[8];
            float x[8];
            if (zstep) {
              ld8(tmem + tm_row + c0, v);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(v[j]) * (kUnZ * kSc);
              if (rowin) put_row8(ZH, ZL, row, c0, ZR, x);
            }
            ld8(tmem + tm_row + L::kTmB + c0, v);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(v[j]) * (kUnZ * kSc);
            if (rowin) put_row8(YH, YL, row, c0, ZR, x);
          }
        }
      } else if (rowwarp) {
        // Final Z^T -> Z^T - 1 1^T / k on the member block, 0 elsewhere (A^-1/2
        // times sqrt(s)); without an operand of its own, P A P / s (from the
        // Gram in TMEM) goes to Y's for the finish.
#pragma unroll 1
        for (int c0 = cb; c0 < ce; c0 += 8) {
          uint32_t v[8];
          ld8(tmem + tm_row + c0, v);
          tmem_wait_ld();
          float x[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int c = c0 + j;
            x[j] = (row < k && c < k) ? __uint_as_float(v[j]) * (kUnZ * kSc) - ik * kSc : 0.0f;
          }
          if (rowin) put_row8(ZH, ZL, row, c0, ZR, x);
          if (!L::kStack) {
            pap8(c0, x);
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] *= is * kSc;
            if (rowin) put_row8(AH, AL, row, c0, ZR, x);
          }
        }
      } else {
        // Warps without rows: X' of the first variables and b -> T rows 0 ..
        // kPre (B operand of E; T is free here).
        for (int vv = (q - NG) * NG + g; vv <= kPre; vv += (4 - NG) * NG) {
          if (vv < kPre && vv >= npre) continue;
          const float* xr = vv < kPre ? V.xpre[vv] : V.b;
          float x[NG];
#pragma unroll
          for (int gg = 0; gg < NG; ++gg) {
            const int m = lane + 32 * gg;
            x[gg] = m < KP ? xr[m] : 0.0f;
          }
          put_x(vv, x);
        }
      }
      if (last) break;
      // P = Z Y (Y as stored), T = a I - b P (scaled step).
      cp_async_wait_all();  // the prefetched X' rows, visible to every thread from the barrier on
      if (!operands_ready(ok)) { alive = false; break; }
      if (warp == 0) {
        tc_fence_after();
        if (elect_one()) {
          h16::issue3<L::kSteps, L::kSlabZ, L::kSlabZ>(tmem, sZH, sZL, sYH, sYL, idescK);
          mma_commit(&mma_bar);
        }
        __syncwarp();
      }
      ns_coeffs(lsp, nsa, nsb);
      const float td = kSc * (nsa - nsb), tb = -kSc * nsb;
      if (!wait_one(&mma_bar, mma_ph)) ok = false;
      mma_ph ^= 1u;
      if (rowwarp) {
        unsigned emax = 0u;  // max |d| by bits: a NaN is above every number
#pragma unroll 1
        for (int c0 = cb; c0 < ce; c0 += 8) {
          uint32_t v[8];
          ld8(tmem + tm_row + c0, v);
          tmem_wait_ld();
          float t[8];
          const int dj = row - c0;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float d = __uint_as_float(v[j]) * kUnZ - ((dj == j) ? 1.0f : 0.0f);
            emax = max(emax, __float_as_uint(d) & 0x7fffffffu);
            t[j] = tb * d + ((dj == j) ? td : 0.0f);  // a I - b P, P = I + d
          }
          if (rowin) put_row8(TH, TL, row, c0, TR, t);
        }
        emax = __reduce_max_sync(0xffffffffu, rowin ? emax : 0u);
        if (lane == 0 && emax >= __float_as_uint(kStop))
          atomicOr(&s_flag[its & 1], emax >= __float_as_uint(kDiverged) ? 3u : 1u);
      }
    }
    if (!alive) break;
    if (diverged) {
      hand_back();
      continue;
    }

    // ---------------- 4. finish ----------------
    // The iterate is Z = p(M) up to rounding errors that the coupled
    // iteration leaves as right factors, so the finish takes C = Z^T A Z:
    // Q^T = Z^T (P A P) (A operand: Z^T rows; B operand: P A P), C^T = Q^T Z;
    // A^-1 = Z C^-1 Z^T, A^-1/2 ~ Z C^-1/2.  The transposed products leave
    // every operand of the next one in the rows that the threads hold (16-byte
    // stores).  E = Z^T [X'^T b] beside Q^T; u = Z^T b is its column kPre.
    if (!operands_ready(ok)) { alive = false; break; }
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
        h16::issue3<L::kSteps, L::kSlabZ, kSlabA>(tmem, sZH, sZL, sAH, sAL, idescK);
        h16::issue3<L::kSteps, L::kSlabZ, L::kSlabT>(tmem + L::kTmE, sZH, sZL, sTH, sTL, idescU);
        mma_commit(&mma_bar);
      }
      __syncwarp();
    }
    if (tid == 0) s_flag[0] = 0u;
    if (!wait_one(&mma_bar, mma_ph)) ok = false;
    mma_ph ^= 1u;
    if (rowwarp) {  // Q^T -> T
#pragma unroll 1
      for (int c0 = cb; c0 < ce; c0 += 8) {
        uint32_t v[8];
        ld8(tmem + tm_row + c0, v);
        tmem_wait_ld();
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __uint_as_float(v[j]) * (kUnZ * kSc);
        if (rowin) put_row8(TH, TL, row, c0, TR, x);
      }
      if (!fast && g == 0) {
        const uint32_t uv = tmem_ld1(tmem + tm_row + L::kTmE + kPre);
        tmem_wait_ld();
        if (rowin) V.u[row] = kUnE * V.xu[kPre] * __uint_as_float(uv);
      }
    }
    // C^T = Q^T Z
    if (!operands_ready(ok)) { alive = false; break; }
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
        h16::issue3<L::kSteps, L::kSlabT, L::kSlabZ>(tmem, sTH, sTL, sZH, sZL, idescK);
        mma_commit(&mma_bar);
      }
      __syncwarp();
    }
    if (!wait_one(&mma_bar, mma_ph)) ok = false;
    mma_ph ^= 1u;
    // F = C - P, symmetric up to rounding (residual).  Short finish: F^T ->
    // Y's operand (A operand of F^T E) and E -> T rows 0 .. 7 (its B operand).
    // Else F^T -> T (B operand of Z F), partial F u, and the rows of Z, read
    // from the columns of Z^T, -> Y's operand (A operand of Z F).
    if (rowwarp) {
      float fu = 0.0f;
      unsigned fm = 0u;  // max |F| by bits: a NaN is above every number
#pragma unroll 1
      for (int c0 = cb; c0 < ce; c0 += 8) {
        uint32_t v[8];
        ld8(tmem + tm_row + c0, v);
        tmem_wait_ld();
        float f[8];
        const int dj = row - c0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int c = c0 + j;
          const float x =
              (row < k && c < k) ? __uint_as_float(v[j]) * kUnZ - (((dj == j) ? 1.0f : 0.0f) - ik) : 0.0f;
          f[j] = x * kScF;
          fm = max(fm, __float_as_uint(x) & 0x7fffffffu);
          if (!fast) fu += x * V.u[c];
        }
        if (rowin && fast) {
          put_row8(YH, YL, row, c0, ZR, f);
        } else if (rowin) {
          put_row8(TH, TL, row, c0, TR, f);
          get_col8(ZH, ZL, row, c0, ZR, f);
          put_row8(YH, YL, row, c0, ZR, f);
        }
      }
      if (fast && g == 0) {
        uint32_t v[8];
        ld8(tmem + tm_row + L::kTmE, v);
        tmem_wait_ld();
        float e8[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) e8[j] = __uint_as_float(v[j]) * (kUnE * kScX);
        if (rowin) put_col8(TH, TL, row, 0, TR, e8);
      }
      if (!fast && rowin) V.part[g][row] = fu;
      fm = __reduce_max_sync(0xffffffffu, rowin ? fm : 0u);
      // NaN or Inf residuals map to the maximum (positive floats order as integers)
      if (lane == 0) atomicMax(&s_flag[0], min(fm, 0x7f800000u));
    }
    // W = cw Z (I - F/2): D = Z F (short finish: D = F^T E, 16 columns)
    if (!operands_ready(ok)) { alive = false; break; }
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
        h16::issue3<L::kSteps, L::kSlabZ, L::kSlabT>(tmem, sYH, sYL, sTH, sTL, fast ? idescU : idescK);
        mma_commit(&mma_bar);
      }
      __syncwarp();
    }
    const float resid = __uint_as_float(s_flag[0]);
    const float c1 = cw * rsqrtf(delta);  // W's eigenvalue on the mean direction
    const float cws = cw * rsqrtf(s);
    if (fast) {  // the mean of X' and sum of X'^2 (one warp per variable)
      for (int vv = warp; vv < prm.n_var; vv += L::kWarps) {
        float sx = 0.0f, sq = 0.0f;
#pragma unroll
        for (int gg = 0; gg < NG; ++gg) {
          const int m = lane + 32 * gg;
          const float x0 = m < KP ? V.xpre[vv][m] : 0.0f;
          sx += x0;
          sq += x0 * x0;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          sx += __shfl_xor_sync(0xffffffffu, sx, off);
          if (rtps) sq += __shfl_xor_sync(0xffffffffu, sq, off);
        }
        if (lane == 0) {
          V.one[vv] = c1 * sx * ik;
          V.xsq[vv] = sq;
          if (prm.Xa32) {
            V.xmh[vv] = (float)V.xmpre[vv];
            V.xml[vv] = (float)(V.xmpre[vv] - (double)V.xmh[vv]);
          }
        }
      }
    } else {
      if (tid < KP) {
        float fu = 0.0f;
#pragma unroll
        for (int gg = 0; gg < NG; ++gg) fu += V.part[gg][tid];
        V.v[tid] = (tid < k) ? V.u[tid] - fu : 0.0f;
      }
      __syncthreads();
      if (tid < KP) {  // wa = c Z v (row tid of Z, in Y's operand)
        float acc = 0.0f;
#pragma unroll 1
        for (int c0 = 0; c0 < KP; c0 += 8) {
          float z[8];
          get_row8(YH, YL, tid, c0, ZR, z);
#pragma unroll
          for (int j = 0; j < 8; ++j) acc += z[j] * V.v[c0 + j];
        }
        V.wa[tid] = sc * is * (1.0f / kSc) * acc;
      }
    }
    if (!wait_all(&mma_bar, mma_ph, ok)) { alive = false; break; }
    mma_ph ^= 1u;
    const bool redo = !conv || !(resid <= fminf(kResidMax, kCondResid * l0));
    if (redo) {
      hand_back();
      continue;
    }
    if (!fast && rowwarp) {  // W rows (over cw / sqrt(s)) -> W^T into Z's operand (A operand of the update)
#pragma unroll 1
      for (int c0 = cb; c0 < ce; c0 += 8) {
        uint32_t v[8];
        ld8(tmem + tm_row + c0, v);
        tmem_wait_ld();
        float w[8];
        get_row8(YH, YL, rowin ? row : 0, c0, ZR, w);
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] -= (0.5f * kUnZF * kSc) * __uint_as_float(v[j]);
        if (rowin) put_col8(ZH, ZL, row, c0, ZR, w);
      }
    }

    // ---------------- 5. update ----------------
    if (fast) {
      // X' W = cw (E - D / 2), D = F^T E, from TMEM; with v = u - F u (column
      // kPre of both) the mean's increment X' wa is c E^T v, a sum over the
      // rows like RTPS's spread.
      const int nv = prm.n_var;
      // Column group g takes the variables g, g + NG, ..
      constexpr int kMine = (kPre + NG - 1) / NG;
      float dv[kMine];
      if (rowwarp) {
        const uint32_t tr = tmem + tm_row;
        uint32_t ev = tmem_ld1(tr + L::kTmE + kPre), uv = tmem_ld1(tr + kPre);
        uint32_t e_[kMine], d_[kMine];
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
          e_[i] = tmem_ld1(tr + L::kTmE + g + i * NG);
          d_[i] = tmem_ld1(tr + g + i * NG);
        }
        tmem_wait_ld();
        const float vr = V.xu[kPre] * (__uint_as_float(ev) * kUnE - kUnD * __uint_as_float(uv));
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
          const int vv = g + i * NG;
          if (vv >= nv) break;
          const bool in = row < k;
          const float e = __uint_as_float(e_[i]) * kUnE;
          dv[i] = in ? cws * V.xu[vv] * (e - 0.5f * kUnD * __uint_as_float(d_[i])) + V.one[vv] : 0.0f;
          float dw = in ? e * vr : 0.0f, s2 = dv[i] * dv[i];
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) {
            dw += __shfl_xor_sync(0xffffffffu, dw, off);
            if (rtps) s2 += __shfl_xor_sync(0xffffffffu, s2, off);
          }
          if (lane == 0) {
            V.sdw[q][vv] = dw;
            V.ssa[q][vv] = s2;
          }
        }
      }
      __syncthreads();
      if (rowwarp && row < k) {
#pragma unroll
        for (int i = 0; i < kMine; ++i) {
          const int vv = g + i * NG;
          if (vv >= nv) break;
          float dw = 0.0f, s2 = 0.0f;
#pragma unroll
          for (int qq = 0; qq < NG; ++qq) {
            dw += V.sdw[qq][vv];
            s2 += V.ssa[qq][vv];
          }
          float a2 = dv[i];
          if (rtps) {
            const float sb = sqrtf(V.xsq[vv] / (float)(k - 1));
            const float sa = sqrtf(s2 / (float)(k - 1));
            a2 *= 1.0f + ((sa > 0.0f) ? (float)prm.rho * (sb - sa) / sa : 0.0f);
          }
          const float inc = sc * is * V.xu[vv] * dw;
          const int64_t o = (base + (int64_t)vv * prm.var_stride) * k + row;
          if (prm.Xa32) prm.Xa32[o] = add3(V.xmh[vv], V.xml[vv], inc, a2);
          else prm.Xa[o] = (V.xmpre[vv] + (double)inc) + (double)a2;
        }
      }
      __syncthreads();
    }
    for (int v0 = 0; !fast && v0 < prm.n_var; v0 += kVarTile) {
      const int nv = (prm.n_var - v0 < kVarTile) ? prm.n_var - v0 : kVarTile;
      // X' rows of the variables -> T rows 0..15 (B operand, K = members);
      // one warp per variable: X' wa, the mean of X', sum of X'^2.
      for (int vv = warp; vv < kVarTile; vv += L::kWarps) {
        const bool pre = v0 == 0 && vv < npre;
        const float* xr = (vv < nv && !pre) ? Xp + (base + (int64_t)(v0 + vv) * prm.var_stride) * k : nullptr;
        float dw = 0.0f, sx = 0.0f, sq = 0.0f, x[NG];
#pragma unroll
        for (int gg = 0; gg < NG; ++gg) {
          const int m = lane + 32 * gg;
          const float x0 = m < KP ? (pre ? V.xpre[vv][m] : ((xr && m < k) ? xr[m] : 0.0f)) : 0.0f;
          x[gg] = x0;
          dw += x0 * (m < KP ? V.wa[m] : 0.0f);
          sx += x0;
          sq += x0 * x0;
        }
        put_x(vv, x);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          dw += __shfl_xor_sync(0xffffffffu, dw, off);
          sx += __shfl_xor_sync(0xffffffffu, sx, off);
          sq += __shfl_xor_sync(0xffffffffu, sq, off);
        }
        if (lane == 0) {
          V.one[vv] = c1 * sx * ik;  // X' W on the mean direction (X' 1 is zero up to rounding)
          V.inc[vv] = dw;
          V.xsq[vv] = sq;
          V.xm[vv] = pre ? V.xmpre[vv] : ((vv < nv) ? prm.xmean[base + (int64_t)(v0 + vv) * prm.var_stride] : 0.0);
        }
      }
      operands_ready(true);
      if (warp == 0) {
        tc_fence_after();
        if (elect_one()) {
          h16::issue3<L::kSteps, L::kSlabZ, L::kSlabT>(tmem, sZH, sZL, sTH, sTL, idescU);
          mma_commit(&mma_bar);
        }
        __syncwarp();
      }
      if (!wait_all(&mma_bar, mma_ph, true)) { alive = false; break; }
      mma_ph ^= 1u;
      float dv[kVarTile];
      if (rowwarp && g == 0) {
        uint32_t v[8], v2[8];
        ld8(tmem + tm_row, v);
        ld8(tmem + tm_row + 8, v2);
        tmem_wait_ld();
#pragma unroll
        for (int vv = 0; vv < 8; ++vv) {
          dv[vv] = cws * kUnE * V.xu[vv] * __uint_as_float(v[vv]) + V.one[vv];
          dv[8 + vv] = cws * kUnE * V.xu[8 + vv] * __uint_as_float(v2[vv]) + V.one[8 + vv];
        }
        if (rtps) {  // analysis spread per variable (members = rows 0 .. KP-1)
#pragma unroll
          for (int vv = 0; vv < kVarTile; ++vv) {
            float s2 = (row < k) ? dv[vv] * dv[vv] : 0.0f;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) s2 += __shfl_xor_sync(0xffffffffu, s2, off);
            if (lane == 0) V.ssa[q][vv] = s2;
          }
        }
      }
      if (rtps) {
        __syncthreads();
        if (tid < kVarTile) {
          float s2 = 0.0f;
#pragma unroll
          for (int qq = 0; qq < NG; ++qq) s2 += V.ssa[qq][tid];
          const float sb = sqrtf(V.xsq[tid] / (float)(k - 1));
          const float sa = sqrtf(s2 / (float)(k - 1));
          V.fac[tid] = (sa > 0.0f) ? (float)prm.rho * (sb - sa) / sa : 0.0f;  // factor - 1
        }
        __syncthreads();
      }
      if (rowwarp && g == 0 && row < k) {
        for (int vv = 0; vv < nv; ++vv) {
          const float a2 = rtps ? dv[vv] * (1.0f + V.fac[vv]) : dv[vv];
          mg::letkf_store(prm, (base + (int64_t)(v0 + vv) * prm.var_stride) * k + row,
                          (V.xm[vv] + (double)V.inc[vv]) + (double)a2);
        }
      }
      __syncthreads();  // T and the vectors are rewritten by the next tile
    }
    if (!alive) break;
    if (tid == 0) {
      atomicAdd(prm.total_local, (unsigned long long)nloc);
      atomicAdd(prm.total_sweeps, (unsigned long long)its);
      atomicMax(prm.max_local, nloc);
      atomicMax(prm.max_sweeps, its);
      atomicMax(prm.max_resid_bits, s_flag[0]);
    }
  }

  if (!alive) {
    // A bounded wait gave up: record it, drain this CTA's MMAs (bounded).
    if (tid == 0) {
      atomicExch(prm.status, 2);
      mma_commit(&mma_bar);
      mbar_wait(&mma_bar, mma_ph);
    }
  }
  cp_async_wait_all();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem, L::kTmemCols);
}

template <int KP>
int launch_tc(const mg::LetkfParams& prm, int num_sms, void* stream, int* ctas) {
  using L = Lay<KP>;
  constexpr size_t kSmem = smem_bytes<KP>();
  auto kern = letkf_tc_kernel<KP>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e != cudaSuccess) return (int)e;
  // The whole unified L1/shared array as shared memory (three KP = 64 CTAs,
  // two of KP = 80 or one of KP = 96 per SM).
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return (int)e;
  // CTAs per SM from the SM's shared memory and register file, at most the
  // design point (which also divides the SM's 512 TMEM columns evenly).
  cudaFuncAttributes fa{};
  e = cudaFuncGetAttributes(&fa, kern);
  if (e != cudaSuccess) return (int)e;
  int dev = 0, smem_sm = 0, reserved = 0, regs_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return (int)e;
  if ((e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev)) != cudaSuccess)
    return (int)e;
  if ((e = cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) != cudaSuccess)
    return (int)e;
  if ((e = cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev)) != cudaSuccess)
    return (int)e;
  const size_t per_cta = kSmem + fa.sharedSizeBytes + (size_t)reserved;
  int per_sm = (int)((size_t)smem_sm / per_cta);
  const int by_regs = fa.numRegs > 0 ? regs_sm / (fa.numRegs * L::kThreads) : L::kMinBlocks;
  if (by_regs < per_sm) per_sm = by_regs;
  if (per_sm > L::kMinBlocks) per_sm = L::kMinBlocks;
  if (per_sm < 1) return (int)cudaErrorInvalidConfiguration;
  int64_t grid = (int64_t)per_sm * num_sms;
  if (grid > prm.npoints) grid = prm.npoints;
  if (grid < 1) grid = 1;
  if (ctas) *ctas = (int)grid;
  kern<<<(unsigned)grid, L::kThreads, kSmem, static_cast<cudaStream_t>(stream)>>>(prm);
  MG_COUNT_LAUNCH();
  return (int)cudaGetLastError();
}

}  // namespace

namespace mg {

bool letkf_tc_supported(const LetkfParams& prm) {
  const bool chol = prm.flags & MG_SQRT_CHOLESKY, upd = prm.flags & MG_UPDATE_COMPAT;
  return prm.k >= 2 && prm.k <= 96 && !chol && !upd && !prm.warm_start && prm.redo_out && prm.n_redo;
}

int letkf_tc_launch(const LetkfParams& prm, int num_sms, void* stream, int* ctas) {
  // The smallest member slots that hold k: fewer slots are less work and more
  // CTAs per SM (k = 80, FP16 pairs: 496 ms in 80 slots; TF32 pairs in 96: 819).
  if (prm.k <= 64) return launch_tc<64>(prm, num_sms, stream, ctas);
  if (prm.k <= 80) return launch_tc<80>(prm, num_sms, stream, ctas);
  return launch_tc<96>(prm, num_sms, stream, ctas);
}

}  // namespace mg
