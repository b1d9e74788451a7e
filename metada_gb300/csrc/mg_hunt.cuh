// FP64 symmetric inverse square root of a k x k SPD matrix by one CTA of 256
// threads, with the eigenvectors found in FP32.
//
// A two-sided FP64 Jacobi needs about ten sweeps of 6 k^3 multiply-adds, and
// GB300 runs two of those per clock per SM.  Instead:
//   1. FP32 Jacobi on A (scaled by a power of four) to a basis V of FP32
//      numbers, made orthonormal to FP32 rounding by one Newton-Schulz step;
//   2. in FP64, D = V^T V - I and B = V^T A V.  Q = V (I + H),
//      H = -D/2 + 3/8 D^2, is orthonormal to FP64 rounding, and
//      A2 = Q^T A Q = B + H B + B H + H B H is diagonal up to E with
//      |E_ij| <= about 1e-5 sqrt(d_i d_j);
//   3. A2^-1/2 = C + F with C = diag(d)^-1/2: the first-order part of F in
//      closed form in FP64, and the fixed point of the remainder
//      (s_i + s_j) G_ij = -[C E F + F E C + F diag(d) F + F E F]_ij, s = sqrt(d),
//      two iterations.
// Every product of two small quantities (H, E, F of order 1e-6) needs only a
// few digits for FP64 accuracy of the result and runs in FP32; FP64 products
// are D, A V and V^T (A V), 2.3 k^3 multiply-adds with their symmetry.
// A^-1/2 = V Ws V^T with Ws = (I + H)(C + F)(I + H), left in two factors.
// A CPU model of this arithmetic against 200-bit references: 6e-16 relative
// at condition number 17, 2e-15 at 300, 6e-14 at 1e4, below LAPACK's FP64
// eigen-solver in each case.  Step 2 shows whether E is small (kHuntGate).
// Where it is not, many eigenvalues are small beside the largest, and the
// FP32 rotations' rounding, eps32 lambda_max, shows between the small ones
// (100 members that span 25 directions well observed: condition number 300).
// A2 is graded by then, and Jacobi on a graded matrix is accurate relative to
// sqrt(d_i d_j): a second pass rotates V on by an FP32 Jacobi of A2 and goes
// back to step 2 with A as the caller kept it.  What is left (or not SPD) goes
// to the caller's FP64 Jacobi.  Two passes end at condition numbers of about a
// million (kHuntMaxCond), as V has FP32 entries: its rounding puts about
// eps32 / 2 sqrt(condition number) into E between the ends of the spectrum.  The
// smallest eigenvalue is known, the prior term's (the mean of the members has
// no obs-space anomaly), and ||A||_F^2 / trace A is a bound of the largest from
// below, so that most systems beyond go back before the first rotation.
#pragma once

#include <cstddef>

#include "mg_dense.cuh"
#include "mg_fp64.cuh"

namespace mg {

constexpr int kHuntThreads = 256;
constexpr float kHuntTol = 1e-5f;   // FP32 Jacobi: off-diagonal threshold relative to sqrt(a_pp a_qq)
constexpr float kHuntGate = 3e-5f;  // largest |E_ij| / sqrt(d_i d_j) accepted
// Condition numbers beyond are not tried (k = 16 .. 100: 1.1e6 passes, 1.5e6
// does not; one pass costs a fifteenth of the FP64 Jacobi, the second as much).
constexpr float kHuntMaxCond = 1.2e6f;

// float -> double by integer operations (conversions run on the FP64 unit);
// FP32 subnormals become zero.
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f);
  const unsigned m = b & 0x7fffffffu;
  if (m < 0x00800000u) return 0.0;
  return __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + (896u << 20))), (int)(b << 29));
}
// The leading 20 bits of a double, as float (small corrections only); zero
// outside FP32's normal range below.
__device__ __forceinline__ float leading(const double* p) {
  const int hi = reinterpret_cast<const int*>(p)[1];
  const int m = hi & 0x7fffffff;
  if (m < (897 << 20)) return 0.0f;
  return __int_as_float((hi & 0x80000000) | ((m - (896 << 20)) << 3));
}

__device__ __forceinline__ int tri(int i, int j) { return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i; }

// The second pass's rotations out of line: inline they take registers from the
// rest of the local kernel (96 members, no second pass: 2.4 % slower) and of
// the global one at 112 slots (2342 against 2320 us), but not at 64 (686
// against 696 us).
template <int KP>
__device__ __noinline__ int jacobi_on(float* A, int lda, float* V, int ldv, int kp, float4* rot) {
  return cta_jacobi_ahead<KP, kHuntThreads, true>(A, lda, V, ldv, kp, kHuntTol, 20, rot);
}

template <int KP>
struct Hunt {
  static constexpr int R = KP / 16;             // 16 x 16 thread grid, R x R elements each
  static constexpr int NL = R * (R + 1) / 2;    // of them in the lower triangle
  static constexpr int LDA = KP + 1, LDV = KP + 4;
  // Regions (bytes): packed FP64 A, then FP32 A / packed FP64 H, V, FP32 F and a block of 16 rows.
  static constexpr int PACKED = KP * (KP + 1) / 2;
  static constexpr size_t A_BYTES = sizeof(double) * PACKED;
  static constexpr size_t B_BYTES = sizeof(double) * PACKED;  // == KP * LDA floats
  static constexpr size_t V_BYTES = sizeof(float) * KP * LDV;
  static constexpr size_t F_BYTES = (sizeof(float) * PACKED + 15) / 16 * 16;
  static constexpr size_t BLK_BYTES = sizeof(double) * 16 * KP;
  static constexpr size_t WORK_BYTES = B_BYTES + V_BYTES + F_BYTES + BLK_BYTES;  // after A
  static constexpr size_t VEC_BYTES = sizeof(double) * 3 * KP + sizeof(float4) * KP + 64;

  double* A;    // in: A (lower rows); out: Ws
  double* H;
  float* A32;
  float* V;     // V[j * LDV + i]: component i of eigenvector j
  float* F;
  double* blk;
  double *d, *s, *c;
  float4* rot;
  int* flag;

  // mem: A_BYTES + WORK_BYTES (16-byte aligned); vec: VEC_BYTES.
  __device__ void carve(unsigned char* a, unsigned char* work, unsigned char* vec) {
    A = reinterpret_cast<double*>(a);
    H = reinterpret_cast<double*>(work);
    A32 = reinterpret_cast<float*>(work);
    V = reinterpret_cast<float*>(work + B_BYTES);
    F = reinterpret_cast<float*>(work + B_BYTES + V_BYTES);
    blk = reinterpret_cast<double*>(work + B_BYTES + V_BYTES + F_BYTES);
    rot = reinterpret_cast<float4*>(vec);
    d = reinterpret_cast<double*>(vec + sizeof(float4) * KP);
    s = d + KP;
    c = s + KP;
    flag = reinterpret_cast<int*>(c + KP);
  }

  // Calls body(u, i, j) for the thread's lower-triangle elements (u static).
  template <typename Fn>
  static __device__ __forceinline__ void lower(int ti, int tj, int k, Fn&& body) {
    int u = 0;
#pragma unroll
    for (int a = 0; a < R; ++a)
#pragma unroll
      for (int b = 0; b <= a; ++b, ++u) {
        const int i = ti + 16 * a, j = tj + 16 * b;
        if (j <= i && i < k) body(u, i, j);
      }
  }

  // t[u] = sum_m X_im Y_mj + Y_im X_mj over symmetric packed X, with
  // Y = Z + diag(w) X / 2 (Z packed, its diagonal left out): the second-order
  // terms of (I + X)(diag + Z)(I + X).
  __device__ void sandwich(float (&t)[NL], const double* X, const double* Z, const double* w, int ti, int tj, int k) {
#pragma unroll
    for (int u = 0; u < NL; ++u) t[u] = 0.0f;
    for (int m = 0; m < k; ++m) {
      const float hw = 0.5f * leading(w + m);
      float xi[R], yi[R], xj[R], yj[R];
#pragma unroll
      for (int a = 0; a < R; ++a) {
        const int i = min(ti + 16 * a, k - 1), j = min(tj + 16 * a, k - 1);
        xi[a] = leading(X + tri(i, m));
        yi[a] = (i == m ? 0.0f : leading(Z + tri(i, m))) + hw * xi[a];
        xj[a] = leading(X + tri(j, m));
        yj[a] = (j == m ? 0.0f : leading(Z + tri(j, m))) + hw * xj[a];
      }
      int u = 0;
#pragma unroll
      for (int a = 0; a < R; ++a)
#pragma unroll
        for (int b = 0; b <= a; ++b, ++u) t[u] += xi[a] * yj[b] + yi[a] * xj[b];
    }
  }

  // A <- Ws with A^-1/2 = scale V Ws V^T.  False: left to the caller (A is
  // destroyed).  All threads; ends synchronised.  prior: the multiple of I in
  // A; reload() fills A as on entry for the second pass.
  template <bool kInline, typename Reload>
  __device__ bool transform(int k, double prior, double* scale, int* sweeps, Reload reload) {
    const int tid = threadIdx.x, ti = tid / 16, tj = tid % 16;
    const int kp = k + (k & 1);
    // ---- scale, FP32 copy, FP32 Jacobi ----
    if (tid == 0) flag[0] = 0;
    __syncthreads();
    for (int i = tid; i < k; i += kHuntThreads) {
      const int ef = (__double2hiint(A[tri(i, i)]) >> 20) & 0x7ff;
      atomicMax(flag, A[tri(i, i)] > 0.0 ? ef : 0x7ff);
    }
    __syncthreads();
    const int ef = flag[0];
    __syncthreads();
    if (ef >= 1900 || ef < 200) return false;  // not positive, not finite or out of range
    const int e2 = (ef - 1023) & ~1;           // A = 2^e2 (entries about 1)
    const double down = __hiloint2double((1023 - e2) << 20, 0);
    *scale = __hiloint2double((1023 - e2 / 2) << 20, 0);
    for (int e = tid; e < KP * LDA; e += kHuntThreads) A32[e] = 0.0f;
    __syncthreads();
    float fro = 0.0f, tr = 0.0f;
    lower(ti, tj, k, [&](int, int i, int j) {
      const double a = A[tri(i, j)] * down;
      A[tri(i, j)] = a;
      const float f = (float)a;
      A32[j * LDA + i] = f;
      fro += (i == j ? 1.0f : 2.0f) * f * f;
      tr += i == j ? f : 0.0f;
    });
    if (tid == 0 && kp > k) A32[k * LDA + k] = 1.0f;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      fro += __shfl_xor_sync(0xffffffffu, fro, off);
      tr += __shfl_xor_sync(0xffffffffu, tr, off);
    }
    if ((tid & 31) == 0) rot[tid >> 5] = make_float4(fro, tr, 0.0f, 0.0f);
    __syncthreads();
    const float most = kHuntMaxCond * (float)(prior * down);  // largest eigenvalue, scaled
    fro = tr = 0.0f;
#pragma unroll
    for (int q = 0; q < kHuntThreads / 32; ++q) {
      fro += rot[q].x;
      tr += rot[q].y;
    }
    if (fro > most * tr) return false;
    *sweeps = cta_jacobi_ahead<KP, kHuntThreads>(A32, LDA, V, LDV, kp, kHuntTol, 20, rot);
    __syncthreads();
    double w[NL];
    float t[NL];
#pragma unroll 1
    for (int pass = 0;; ++pass) {
      // ---- V <- (3 I - V V^T) V / 2 (rows are eigenvectors), in FP32 ----
      {
        float* M = A32;
        float acc[R][R];
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
          for (int b = 0; b < R; ++b) acc[a][b] = 0.0f;
        for (int m = 0; m < KP; m += 4) {
          float4 x[R], y[R];
#pragma unroll
          for (int a = 0; a < R; ++a) {
            const int i = ti + 16 * a, j = tj + 16 * a;
            x[a] = (i < k && m < kp) ? *reinterpret_cast<const float4*>(V + i * LDV + m) : make_float4(0, 0, 0, 0);
            y[a] = (j < k && m < kp) ? *reinterpret_cast<const float4*>(V + j * LDV + m) : make_float4(0, 0, 0, 0);
          }
#pragma unroll
          for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b < R; ++b)
              acc[a][b] += (x[a].x * y[b].x + x[a].y * y[b].y) + (x[a].z * y[b].z + x[a].w * y[b].w);
        }
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
          for (int b = 0; b < R; ++b) {
            const int i = ti + 16 * a, j = tj + 16 * b;
            M[i * LDA + j] = (i == j ? 1.5f : 0.0f) - 0.5f * acc[a][b];
            acc[a][b] = 0.0f;
          }
        __syncthreads();
        for (int m = 0; m < k; ++m) {
          float x[R], y[R];
#pragma unroll
          for (int a = 0; a < R; ++a) {
            x[a] = M[(ti + 16 * a) * LDA + m];
            y[a] = V[m * LDV + tj + 16 * a];
          }
#pragma unroll
          for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b < R; ++b) acc[a][b] += x[a] * y[b];
        }
        __syncthreads();
#pragma unroll
        for (int a = 0; a < R; ++a)
#pragma unroll
          for (int b = 0; b < R; ++b) {
            const int i = ti + 16 * a, j = tj + 16 * b;
            if (i < k) V[i * LDV + j] = j < k ? acc[a][b] : 0.0f;  // beyond k: zero, read in fours below
          }
        __syncthreads();
      }
      // ---- H = -D/2 + 3/8 D^2, D = V V^T - I in FP64 ----
#pragma unroll
      for (int u = 0; u < NL; ++u) w[u] = 0.0;
      for (int m = 0; m < k; m += 4) {
        float4 x[R], y[R];
#pragma unroll
        for (int a = 0; a < R; ++a) {
          x[a] = *reinterpret_cast<const float4*>(V + min(ti + 16 * a, k - 1) * LDV + m);
          y[a] = *reinterpret_cast<const float4*>(V + min(tj + 16 * a, k - 1) * LDV + m);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double xd[R], yd[R];
#pragma unroll
          for (int a = 0; a < R; ++a) {
            xd[a] = widen(q == 0 ? x[a].x : (q == 1 ? x[a].y : (q == 2 ? x[a].z : x[a].w)));
            yd[a] = widen(q == 0 ? y[a].x : (q == 1 ? y[a].y : (q == 2 ? y[a].z : y[a].w)));
          }
          int u = 0;
#pragma unroll
          for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b, ++u) w[u] = __fma_rn(xd[a], yd[b], w[u]);
        }
      }
      lower(ti, tj, k, [&](int u, int i, int j) { H[tri(i, j)] = w[u] - (i == j ? 1.0 : 0.0); });
      __syncthreads();
      {
        float t[NL];
#pragma unroll
        for (int u = 0; u < NL; ++u) t[u] = 0.0f;
        for (int m = 0; m < k; ++m) {
          float xi[R], xj[R];
#pragma unroll
          for (int a = 0; a < R; ++a) {
            xi[a] = leading(H + tri(min(ti + 16 * a, k - 1), m));
            xj[a] = leading(H + tri(min(tj + 16 * a, k - 1), m));
          }
          int u = 0;
#pragma unroll
          for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b, ++u) t[u] += xi[a] * xj[b];
        }
        __syncthreads();
        lower(ti, tj, k, [&](int u, int i, int j) {
          H[tri(i, j)] = __fma_rn(-0.5, H[tri(i, j)], widen(0.375f * t[u]));
        });
      }
      // ---- B = V A V^T (rows of V), in blocks of 16 rows of A ----
#pragma unroll
      for (int u = 0; u < NL; ++u) w[u] = 0.0;
      for (int mb = 0; mb < k; mb += 16) {
        {
          const int m = min(mb + ti, k - 1);
          double p[R];
#pragma unroll
          for (int b = 0; b < R; ++b) p[b] = 0.0;
          for (int l = 0; l < k; l += 4) {
            float4 y[R];
#pragma unroll
            for (int b = 0; b < R; ++b) y[b] = *reinterpret_cast<const float4*>(V + min(tj + 16 * b, k - 1) * LDV + l);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (l + q >= k) break;
              const double a = A[tri(m, l + q)];
#pragma unroll
              for (int b = 0; b < R; ++b)
                p[b] = __fma_rn(a, widen(q == 0 ? y[b].x : (q == 1 ? y[b].y : (q == 2 ? y[b].z : y[b].w))), p[b]);
            }
          }
#pragma unroll
          for (int b = 0; b < R; ++b) blk[ti * KP + tj + 16 * b] = p[b];
        }
        __syncthreads();
        for (int m = 0; m < 16 && mb + m < k; ++m) {
          double x[R], y[R];
#pragma unroll
          for (int a = 0; a < R; ++a) {
            x[a] = widen(V[min(ti + 16 * a, k - 1) * LDV + mb + m]);
            y[a] = blk[m * KP + tj + 16 * a];
          }
          int u = 0;
#pragma unroll
          for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b, ++u) w[u] = __fma_rn(x[a], y[b], w[u]);
        }
        __syncthreads();
      }
      // ---- A2 = (I + H) B (I + H) = diag(d) + E ----
      lower(ti, tj, k, [&](int u, int i, int j) {
        A[tri(i, j)] = w[u];
        if (i == j) d[i] = w[u];
      });
      if (tid == 0) flag[0] = flag[1] = 0;
      __syncthreads();
      sandwich(t, H, A, d, ti, tj, k);
      lower(ti, tj, k, [&](int u, int i, int j) { w[u] += __fma_rn(H[tri(i, j)], d[i] + d[j], widen(t[u])); });
      __syncthreads();
      lower(ti, tj, k, [&](int u, int i, int j) {
        A[tri(i, j)] = w[u];
        if (i == j) {
          const double dd = w[u], sq = sqrt(dd);
          d[i] = dd;
          s[i] = sq;
          c[i] = 1.0 / sq;
          if (!(dd > 0.0)) flag[0] = 1;
        }
      });
      __syncthreads();
      // ---- F = F1 + G; w: F1, t: G ----
      lower(ti, tj, k, [&](int u, int i, int j) {
        t[u] = 0.0f;
        if (i == j) {
          w[u] = 0.0;
          return;
        }
        const float e = leading(A + tri(i, j)) * leading(c + i) * leading(c + j);
        if (!(fabsf(e) <= kHuntGate)) flag[1] = 1;
        const double si = s[i], sj = s[j];
        w[u] = -w[u] * recip_fp64(si * sj * (si + sj));
      });
      __syncthreads();
      if (flag[0]) return false;
      if (!flag[1]) break;
      if (pass > 0) return false;
      float top = 0.0f;
      for (int i = 0; i < k; ++i) top = fmaxf(top, leading(d + i));
      if (top > most) return false;
      for (int e = tid; e < KP * LDA; e += kHuntThreads) A32[e] = 0.0f;
      __syncthreads();
      lower(ti, tj, k, [&](int, int i, int j) { A32[j * LDA + i] = (float)A[tri(i, j)]; });
      if (tid == 0 && kp > k) A32[k * LDA + k] = 1.0f;
      __syncthreads();
      if constexpr (kInline) *sweeps += cta_jacobi_ahead<KP, kHuntThreads, true>(A32, LDA, V, LDV, kp, kHuntTol, 20, rot);
      else *sweeps += jacobi_on<KP>(A32, LDA, V, LDV, kp, rot);
      __syncthreads();
      reload();
      __syncthreads();
      lower(ti, tj, k, [&](int, int i, int j) { A[tri(i, j)] *= down; });
      __syncthreads();
    }
    float* T1 = reinterpret_cast<float*>(blk);
#pragma unroll 1
    for (int it = 0; it < 2; ++it) {
      lower(ti, tj, k, [&](int u, int i, int j) { F[tri(i, j)] = (float)w[u] + t[u]; });
      __syncthreads();
#pragma unroll
      for (int u = 0; u < NL; ++u) t[u] = 0.0f;
#pragma unroll
      for (int mb = 0; mb < R; ++mb) {
        if (16 * mb < k) {
          const int m = min(16 * mb + ti, k - 1);
          float p[R];
#pragma unroll
          for (int b = 0; b < R; ++b) p[b] = 0.0f;
          for (int l = 0; l < k; ++l) {
            const float e = l == m ? 0.0f : leading(A + tri(m, l));
#pragma unroll
            for (int b = 0; b < R; ++b) p[b] += e * F[tri(l, min(tj + 16 * b, k - 1))];
          }
#pragma unroll
          for (int b = 0; b < R; ++b) T1[ti * KP + tj + 16 * b] = p[b];
        }
        __syncthreads();
        if (16 * mb < k) {
          for (int m = 0; m < 16 && 16 * mb + m < k; ++m) {
            const int gm = 16 * mb + m;
            const float dm = leading(d + gm);
            float x[R], y[R];
#pragma unroll
            for (int a = 0; a < R; ++a) {
              const int j = min(tj + 16 * a, k - 1);
              x[a] = F[tri(min(ti + 16 * a, k - 1), gm)];
              y[a] = dm * F[tri(gm, j)] + T1[m * KP + j];
            }
            int u = 0;
#pragma unroll
            for (int a = 0; a < R; ++a)
#pragma unroll
              for (int b = 0; b <= a; ++b, ++u) t[u] += x[a] * y[b];
          }
          int u = 0;
#pragma unroll
          for (int a = 0; a < R; ++a)
#pragma unroll
            for (int b = 0; b <= a; ++b, ++u) {
              const int i = min(ti + 16 * a, k - 1), j = min(tj + 16 * b, k - 1);
              if (a == mb) t[u] += leading(c + i) * T1[(i - 16 * mb) * KP + j];
              if (b == mb) t[u] += leading(c + j) * T1[(j - 16 * mb) * KP + i];
            }
        }
        __syncthreads();
      }
      lower(ti, tj, k, [&](int u, int i, int j) { t[u] = -t[u] / (leading(s + i) + leading(s + j)); });
    }
    // ---- Ws = (I + H)(C + F)(I + H) ----
    lower(ti, tj, k, [&](int u, int i, int j) {
      w[u] += widen(t[u]);
      if (i == j) w[u] += c[i];
      A[tri(i, j)] = w[u];
    });
    __syncthreads();
    sandwich(t, H, A, c, ti, tj, k);
    lower(ti, tj, k, [&](int u, int i, int j) { w[u] += __fma_rn(H[tri(i, j)], c[i] + c[j], widen(t[u])); });
    __syncthreads();
    lower(ti, tj, k, [&](int u, int i, int j) { A[tri(i, j)] = w[u]; });
    __syncthreads();
    return true;
  }

  // Y_r = V Ws V^T X_r for nr rows of length k (stride KP); T is scratch of
  // the same size, X is overwritten.  Ends synchronised.
  __device__ void apply(double* X, double* T, double* Y, int nr, int k) {
    const int tid = threadIdx.x;
    for (int e = tid; e < nr * k; e += kHuntThreads) {
      const int r = e / k, j = e - r * k;
      double a = 0.0;
      for (int m = 0; m < k; m += 4) {
        const float4 v = *reinterpret_cast<const float4*>(V + j * LDV + m);
        a = __fma_rn(X[r * KP + m], widen(v.x), a);
        if (m + 1 < k) a = __fma_rn(X[r * KP + m + 1], widen(v.y), a);
        if (m + 2 < k) a = __fma_rn(X[r * KP + m + 2], widen(v.z), a);
        if (m + 3 < k) a = __fma_rn(X[r * KP + m + 3], widen(v.w), a);
      }
      T[r * KP + j] = a;
    }
    __syncthreads();
    for (int e = tid; e < nr * k; e += kHuntThreads) {
      const int r = e / k, i = e - r * k;
      double a = 0.0;
      for (int j = 0; j < k; ++j) a = __fma_rn(A[tri(i, j)], T[r * KP + j], a);
      X[r * KP + i] = a;
    }
    __syncthreads();
    for (int e = tid; e < nr * k; e += kHuntThreads) {
      const int r = e / k, m = e - r * k;
      double a = 0.0;
      for (int j = 0; j < k; ++j) a = __fma_rn(X[r * KP + j], widen(V[j * LDV + m]), a);
      Y[r * KP + m] = a;
    }
    __syncthreads();
  }
};

}  // namespace mg
