// FP64 products on the tensor cores by exact splitting (the error-free
// transformation of Ozaki, Ogita, Oishi and Rump, 2012).
//
// GB300 runs two FP64 multiply-adds per clock per SM, its tensor cores about
// a thousand FP16 ones through mma.sync.  An operand's rows (along the
// contraction) are scaled by a power of two and rounded to 55-bit integers,
// which are seven balanced base-256 digits (-128 .. 127, the bytes of
// x + 0x80808080808080); the products of digit slices s and t are integers
// whose sums over up to 112 terms stay below 2^24, so FP32 accumulation is
// exact, and the slices with s + t <= 6 (28 of 49) leave out less than
// 2^-54 of (largest |a|) (largest |b|) per term: FP64 rounding.  mma.sync
// and not tcgen05: the digits of one tile are produced by the threads that
// consume them and an accumulator set is 28 registers.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace mg {
namespace oz {

constexpr int kSlices = 7;

// Exponent field of |v| (0 for zeros and subnormals).
__device__ __forceinline__ int ef_of(double v) { return (__double2hiint(v) >> 20) & 0x7ff; }

// round(v 2^(54 - ex)) for |v| < 2^ex, ex = efmax - 1022, efmax >= 1: |result| <= 2^54.
__device__ __forceinline__ long long to_fixed(double v, int efmax) {
  const long long b = __double_as_longlong(v);
  const int ef = (int)(b >> 52) & 0x7ff;
  const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | (ef ? 1ull << 52 : 0ull);
  int r = efmax - (ef ? ef : 1);
  r = r < 0 ? 0 : (r > 60 ? 60 : r);
  const unsigned long long h = r ? 1ull << (r - 1) : 0ull;
  const long long x = (long long)(((m << 1) + h) >> r);
  return b < 0 ? -x : x;
}

// Digit slices of eight values (contiguous along the contraction): slice s
// (0 the most significant) as eight halves at dst + s * stride (16-byte
// aligned).
__device__ __forceinline__ void store_digits8(const double (&v)[8], int efmax, __half* dst, int stride) {
  unsigned lo[8], hi[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const unsigned long long u = (unsigned long long)(to_fixed(v[q], efmax) + 0x0080808080808080ll);
    lo[q] = (unsigned)u;
    hi[q] = (unsigned)(u >> 32);
  }
  const __half2 c1152 = __half2half2(__ushort_as_half((unsigned short)0x6480));
#pragma unroll
  for (int s = 0; s < kSlices; ++s) {
    const int t = kSlices - 1 - s;  // byte of u
    const unsigned pick = (t & 3) | ((4 + (t & 3)) << 4);
    uint4 w;
    unsigned* wp = reinterpret_cast<unsigned*>(&w);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      // halves 1024 + byte, then minus 1152: exact
      const unsigned two = __byte_perm(t < 4 ? lo[2 * q] : hi[2 * q], t < 4 ? lo[2 * q + 1] : hi[2 * q + 1], pick);
      const unsigned bits = __byte_perm(two, 0x64646464u, 0x4140);
      const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&bits), c1152);
      wp[q] = *reinterpret_cast<const unsigned*>(&h);
    }
    *reinterpret_cast<uint4*>(dst + s * stride) = w;
  }
}

__device__ __forceinline__ void ldsm4(unsigned (&r)[4], const __half* p) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void ldsm2(unsigned (&r)[2], const __half* p) {
  const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(p));
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// One 16 x 8 output tile over KS k-steps of 16: acc[d] = sum over s + t = d
// of A_s B_t.  A: rows of the tile at a (row stride lda halves, slices sa
// apart), B: columns of the tile at b, both contiguous along the contraction.
template <int KS>
__device__ __forceinline__ void tile(float (&acc)[kSlices][4], const __half* a, int lda, int sa, const __half* b,
                                     int ldb, int sb) {
  const int lane = threadIdx.x & 31;
  const __half* ap = a + (lane & 15) * lda + (lane >> 4) * 8;
  const __half* bp = b + (lane & 7) * ldb + ((lane >> 3) & 1) * 8;
#pragma unroll
  for (int d = 0; d < kSlices; ++d)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[d][e] = 0.0f;
#pragma unroll 1
  for (int ks = 0; ks < KS; ++ks) {
    unsigned bf[kSlices][2];
#pragma unroll
    for (int t = 0; t < kSlices; ++t) ldsm2(bf[t], bp + t * sb + ks * 16);
#pragma unroll
    for (int s = 0; s < kSlices; ++s) {
      unsigned af[4];
      ldsm4(af, ap + s * sa + ks * 16);
#pragma unroll
      for (int t = 0; t < kSlices - s; ++t) mma(acc[s + t], af, bf[t]);
    }
  }
}

// Entry e of the tile's sum as an integer in units of 2^52 of the product of
// the two fixed-point scales (|result| < 2^63 for up to 112 terms).
__device__ __forceinline__ long long combine(const float (&acc)[kSlices][4], int e) {
  const int p1 = (int)acc[0][e] * 256 + (int)acc[1][e];
  const int p2 = (int)acc[2][e] * 256 + (int)acc[3][e];
  const int p3 = (int)acc[4][e] * 256 + (int)acc[5][e];
  const long long t = ((long long)p1 << 32) + ((long long)p2 << 16) + p3;
  return t * 16 + ((int)acc[6][e] >> 4);
}

// 2^(exa + exb - 56), the weight of combine()'s unit for operand exponents
// fields ea, eb (2^ex = 2^(ef - 1022)); zero below the normal range, up to a
// sum of kUnitEf (products below 2^-968: nothing beside a Gram's k - 1).
constexpr int kUnitEf = 1077;
__device__ __forceinline__ double unit(int ea, int eb) {
  const int f = ea + eb - kUnitEf;
  return f > 0 ? __hiloint2double(f << 20, 0) : 0.0;
}
// Exponent fields up to which unit() and the scaled sums stay finite.
constexpr int kMaxEf = 1500;

}  // namespace oz
}  // namespace mg
