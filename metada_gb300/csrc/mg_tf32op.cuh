// TF32 tensor-core operands in shared memory: K-major with the 128-byte
// swizzle (a slab holds 32 TF32 columns of all its rows, 128 bytes per row,
// 8-row groups 1024 bytes apart), each value kept as a hi and a lo part (hi =
// x rounded to TF32, lo = x - hi).  The Gram of the tensor-core local analyses
// (mg_letkf_tc.cu), whose obs rows need FP32's exponent range; FP16 pairs
// (mg_f16op.cuh) take half the space.
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

// D (TMEM) (+)= A B^T over one slab of 32 K-columns (4 K-steps of 8).  A: 128
// rows; B: N rows.  Called by one thread.
static __device__ __forceinline__ void issue_slab(uint32_t dtm, uint32_t a, uint32_t b, uint32_t idesc,
                                                  bool accumulate) {
  // Descriptors of the first K-step; later steps add (byte offset >> 4) to
  // the 14-bit start-address field (shared addresses stay below 256 KB).
  const uint64_t ad = smem_desc_sw128(a), bd = smem_desc_sw128(b);
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    const uint64_t o = (uint64_t)(kk * 32 >> 4);
    mma_tf32(dtm, ad + o, bd + o, idesc, (accumulate || kk > 0) ? 1u : 0u);
  }
}

// Operands written by the generic proxy become visible to the tensor core,
// earlier TMEM reads are ordered before what follows the barrier.  One
// CTA-wide decision on the waits of the step before: false if any thread's
// gave up.
static __device__ __forceinline__ bool operands_ready(bool ok) {
  fence_proxy_async_smem();
  tc_fence_before();
  return __syncthreads_or(ok ? 0 : 1) == 0;
}

// This thread waits (bounded) for the phase; what it reads or writes next is
// in bounds either way, and operands_ready takes the CTA's decision.  The poll
// runs per lane: the warp comes together before its tensor-memory loads.
static __device__ __forceinline__ bool wait_one(uint64_t* bar, uint32_t parity) {
  const bool ok = mbar_wait(bar, parity);
  __syncwarp();
  tc_fence_after();
  return ok;
}

// As wait_one, with the CTA's decision at once.
static __device__ __forceinline__ bool wait_all(uint64_t* bar, uint32_t parity, bool ok) {
  if (!mbar_wait(bar, parity)) ok = false;
  const int bad = __syncthreads_or(ok ? 0 : 1);
  tc_fence_after();
  return bad == 0;
}

}  // namespace t5
}  // namespace mg
