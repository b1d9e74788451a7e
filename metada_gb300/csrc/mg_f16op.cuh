// FP16 tensor-core operands in shared memory and the 3-pass product:
// K-major operands with the 64-byte swizzle (a slab holds 32 columns of all
// its rows, 64 bytes per row, 8-row groups 512 bytes apart), each value
// stored as a hi and a lo copy (hi = x rounded to FP16, lo = x - hi rounded
// to FP16: 22 significant bits together, as the TF32 split of mg_tf32op.cuh
// gives), and D += A B^T issued as hi*hi + hi*lo + lo*hi per K-step of 16,
// accumulated in FP32.  Against TF32 operands: half the shared memory and
// stores, half the MMA time.  FP16's range is the caller's: values are
// handed over multiplied by a power of two that keeps them below 65504 and
// the lo copies' subnormal floor (2^-25) below FP32 rounding of the largest.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "mg_tcgen05.cuh"

namespace mg {
namespace t5 {
namespace h16 {

// Byte offset of element (row r, column c) in an operand whose slabs (32
// columns each) hold `rows` rows.
static __device__ __forceinline__ uint32_t off(int r, int c, uint32_t rows) {
  return (uint32_t)(c >> 5) * rows * 64u + (uint32_t)r * 64u +
         ((uint32_t)(((c & 31) >> 3) ^ ((r >> 1) & 3)) << 4) + (uint32_t)(c & 7) * 2u;
}

static __device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Row r, columns c0 .. c0+7 (c0 a multiple of 8): one 16-byte chunk each
// (conflict-free across a warp's 32 consecutive rows).
static __device__ __forceinline__ void put_row8(unsigned char* hi, unsigned char* lo, int r, int c0, uint32_t rows,
                                                const float (&x)[8]) {
  uint4 vh, vl;
  split2(x[0], x[1], vh.x, vl.x);
  split2(x[2], x[3], vh.y, vl.y);
  split2(x[4], x[5], vh.z, vl.z);
  split2(x[6], x[7], vh.w, vl.w);
  const uint32_t o = off(r, c0, rows);
  *reinterpret_cast<uint4*>(hi + o) = vh;
  *reinterpret_cast<uint4*>(lo + o) = vl;
}

// The same values to two operands.
static __device__ __forceinline__ void put_row8x2(unsigned char* hi, unsigned char* lo, uint32_t rows,
                                                  unsigned char* hi2, unsigned char* lo2, uint32_t rows2, int r, int c0,
                                                  const float (&x)[8]) {
  uint4 vh, vl;
  split2(x[0], x[1], vh.x, vl.x);
  split2(x[2], x[3], vh.y, vl.y);
  split2(x[4], x[5], vh.z, vl.z);
  split2(x[6], x[7], vh.w, vl.w);
  const uint32_t o = off(r, c0, rows), o2 = off(r, c0, rows2);
  *reinterpret_cast<uint4*>(hi + o) = vh;
  *reinterpret_cast<uint4*>(lo + o) = vl;
  *reinterpret_cast<uint4*>(hi2 + o2) = vh;
  *reinterpret_cast<uint4*>(lo2 + o2) = vl;
}

static __device__ __forceinline__ void get_row8(const unsigned char* hi, const unsigned char* lo, int r, int c0,
                                                uint32_t rows, float (&x)[8]) {
  const uint32_t o = off(r, c0, rows);
  const uint4 vh = *reinterpret_cast<const uint4*>(hi + o), vl = *reinterpret_cast<const uint4*>(lo + o);
  const uint32_t h[4] = {vh.x, vh.y, vh.z, vh.w}, l[4] = {vl.x, vl.y, vl.z, vl.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&h[j]));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&l[j]));
    x[2 * j] = a.x + b.x;
    x[2 * j + 1] = a.y + b.y;
  }
}

// Transposed: the thread's row kk of a matrix, columns n0 .. n0+7, goes to
// operand rows n0 .. n0+7 at column kk (2-byte stores; a warp's 32
// consecutive kk fill one 64-byte row).
static __device__ __forceinline__ void put_col8(unsigned char* hi, unsigned char* lo, int kk, int n0, uint32_t rows,
                                                const float (&x)[8]) {
  const uint32_t cb = (uint32_t)(kk >> 5) * rows * 64u + (uint32_t)(kk & 7) * 2u + (uint32_t)n0 * 64u;
  const int ch = (kk & 31) >> 3;
#pragma unroll
  for (int j = 0; j < 8; j += 2) {  // n0 is a multiple of 8: rows n0 + j and n0 + j + 1 share a swizzle phase
    uint32_t h, l;
    split2(x[j], x[j + 1], h, l);
    const uint32_t o = cb + (uint32_t)j * 64u + ((uint32_t)(ch ^ (j >> 1)) << 4);
    *reinterpret_cast<uint16_t*>(hi + o) = (uint16_t)h;
    *reinterpret_cast<uint16_t*>(lo + o) = (uint16_t)l;
    *reinterpret_cast<uint16_t*>(hi + o + 64) = (uint16_t)(h >> 16);
    *reinterpret_cast<uint16_t*>(lo + o + 64) = (uint16_t)(l >> 16);
  }
}

static __device__ __forceinline__ void get_col8(const unsigned char* hi, const unsigned char* lo, int c, int r0,
                                                uint32_t rows, float (&x)[8]) {
  const uint32_t cb = (uint32_t)(c >> 5) * rows * 64u + (uint32_t)(c & 7) * 2u + (uint32_t)r0 * 64u;
  const int ch = (c & 31) >> 3;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t o = cb + (uint32_t)j * 64u + ((uint32_t)(ch ^ (j >> 1)) << 4);
    x[j] = __half2float(*reinterpret_cast<const __half*>(hi + o)) +
           __half2float(*reinterpret_cast<const __half*>(lo + o));
  }
}

// SWIZZLE_64B, K-major: rows of 64 bytes, 8-row groups 512 bytes apart.
static __device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);        // start address
  d |= (uint64_t)1 << 16;                        // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)((512 >> 4) & 0x3FFF) << 32;    // stride byte offset
  d |= (uint64_t)1 << 46;                        // descriptor version (SM100)
  d |= (uint64_t)4 << 61;                        // layout: SWIZZLE_64B
  return d;
}

// kind::f16 with FP16 operands (format 0), D = F32, both K-major.
__host__ __device__ constexpr uint32_t idesc_f16_f32(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

static __device__ __forceinline__ void mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// D (TMEM) = A B over NK K-steps of 16, 3 passes each.  A: 128 rows from
// a_hi / a_lo (slab stride A_SLAB); B: N rows from b_hi / b_lo.  Called by one
// thread.  Unrolled and inline: the descriptors are constants off the
// operands' addresses; as a loop in a function of its own, the issue took
// 1300 cycles of a step in which the tensor core needs about 500.
template <int NK, uint32_t A_SLAB, uint32_t B_SLAB>
static __device__ __forceinline__ void issue3(uint32_t dtm, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi, uint32_t b_lo,
                                              uint32_t idesc) {
  const uint64_t ah = smem_desc_sw64(a_hi), al = smem_desc_sw64(a_lo);
  const uint64_t bh = smem_desc_sw64(b_hi), bl = smem_desc_sw64(b_lo);
#pragma unroll
  for (int s = 0; s < NK; ++s) {
    const uint64_t ao = (uint64_t)(((s >> 1) * A_SLAB + (s & 1) * 32) >> 4);
    const uint64_t bo = (uint64_t)(((s >> 1) * B_SLAB + (s & 1) * 32) >> 4);
    mma(dtm, ah + ao, bh + bo, idesc, s > 0 ? 1u : 0u);
    mma(dtm, ah + ao, bl + bo, idesc, 1u);
    mma(dtm, al + ao, bh + bo, idesc, 1u);
  }
}

}  // namespace h16
}  // namespace t5
}  // namespace mg
