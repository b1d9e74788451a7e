// TF32 tensor-core operands in shared memory and the 3-pass product:
// K-major operands with the 128-byte swizzle (a slab holds 32 TF32 columns
// of all its rows, 128 bytes per row, 8-row groups 1024 bytes apart), each
// value stored as a hi and a lo copy (hi = x rounded to TF32, lo = x - hi),
// and D += A B^T issued as hi*hi + hi*lo + lo*hi per K-step of 8.  The
// Gram of the tensor-core local analyses (mg_letkf_tc.cu), whose obs rows
// need FP32's exponent range; FP16 pairs (mg_f16op.cuh) take half the space.
#pragma once

#include <stdint.h>

#include "mg_tcgen05.cuh"

namespace mg {
namespace t5 {

// ---- operand addressing: K-major, 128-byte swizzle, TF32 in 32-bit words ----
// Byte offset of element (row r, column c) in an operand whose slabs (32
// columns each) hold `rows` rows.
static __device__ __forceinline__ uint32_t sw_off(int r, int c, uint32_t rows) {
  return (uint32_t)(c >> 5) * rows * 128u + (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u +
         ((uint32_t)(((c & 31) >> 2) ^ (r & 7)) << 4) + (uint32_t)(c & 3) * 4u;
}

static __device__ __forceinline__ void split(float x, float& h, float& l) {
  h = tf32_rna(x);
  l = x - h;
}

// D (TMEM) += A B over nslab slabs of 32 K-columns, 3 passes per K-step of 8.
// A: 128 rows from a_hi/a_lo (slab stride a_slab); B: N rows from b_hi/b_lo.
// Called by all of warp 0 with the same arguments (lane 0 issues); out of
// line: one copy of the issue loop for every product of the kernel.
static __device__ __noinline__ void issue3(uint32_t dtm, uint32_t a_hi, uint32_t a_lo, uint32_t a_slab, uint32_t b_hi,
                                       uint32_t b_lo, uint32_t b_slab, int nslab, uint32_t idesc, bool accumulate) {
  // Descriptors of the first K-step; later steps add (byte offset >> 4) to
  // the 14-bit start-address field (shared addresses stay below 256 KB).
  const uint64_t ah = smem_desc_sw128(a_hi), al = smem_desc_sw128(a_lo);
  const uint64_t bh = smem_desc_sw128(b_hi), bl = smem_desc_sw128(b_lo);
  for (int s = 0; s < nslab; ++s) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const uint64_t ao = (uint64_t)((s * a_slab + kk * 32) >> 4), bo = (uint64_t)((s * b_slab + kk * 32) >> 4);
      mma_tf32_elect(dtm, ah + ao, bh + bo, idesc, (accumulate || s > 0 || kk > 0) ? 1u : 0u);
      mma_tf32_elect(dtm, ah + ao, bl + bo, idesc, 1u);
      mma_tf32_elect(dtm, al + ao, bh + bo, idesc, 1u);
    }
  }
}

// Operands written by the generic proxy become visible to the tensor core,
// earlier TMEM reads are ordered before what follows the barrier.
static __device__ __forceinline__ void operands_ready() {
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
}

// Every thread waits (bounded) for the phase; one CTA-wide decision.
static __device__ __forceinline__ bool wait_all(uint64_t* bar, uint32_t parity) {
  const bool ok = mbar_wait(bar, parity);
  const int bad = __syncthreads_or(ok ? 0 : 1);
  tc_fence_after();
  return bad == 0;
}

}  // namespace t5
}  // namespace mg
