// local_update.cuh — tet and triangle local updates for the GB300 FIM kernels.
//
// The arithmetic reproduces the reference updates bit for bit:
//   tet:      localSolverTet1, src/core3d/cuda/CUDA_kernels.cu:69-225
//   triangle: inline update in FIMCuda, src/core2d/cuda/CUDA_kernels.cu:143-204
// Every expression keeps the reference's association and operand order, because
// nvcc's multiply-add contraction (on by default, as in the reference build) pairs
// products with sums by position; the same expression trees give the same fused
// roundings.
//
// The reference divides in FP64 in two places: `(-q ± sqrt(delta)) / (2.0*p)` and
// `(s*lambda1 + t) / (h + 1e-8)` (the 2.0 and the 1e-8 literal are doubles).  GB300
// runs FP64 at 1/64 of the FP32 rate, so this file computes both quotients in FP32
// with the same final bits:
//   * root_quot: an IEEE float division by 2p.  For float operands a double
//     quotient rounded to float equals the correctly rounded float quotient
//     (53 >= 2*24 + 2, the innocuous double rounding bound), so the only cases left
//     are |p| so large that 2p overflows in float; those take the FP64 path.
//   * small_quot: the denominator h + 1e-8 is carried as an unevaluated float pair,
//     the quotient is corrected with an exact FMA residual, and the result is
//     accepted only when it lies clearly away from a rounding boundary; otherwise
//     (about once in a million calls) the FP64 division runs.
#pragma once

#include <cuda_runtime.h>

namespace eikgb {

constexpr float kLarge3DDev = 1000000000.0f;
constexpr float kLarge2DDev = 10000000.0f;

// Rare paths (FP64 divisions) and the whole of small_quot stay out of line: the
// four inlined tet updates of a slot are large, and moving code that runs once in
// a million calls out of them cuts instruction-cache misses (the sweep kernels ran
// 10% faster on a 65^3 cube, same bits).  Calls do not change the arithmetic.
__device__ __noinline__ float root_quot_slow(float num, float p) {
  return (float)((double)num / (2.0 * (double)p));
}

__device__ __forceinline__ float root_quot(float num, float p) {
  if (fabsf(p) < 0x1p126f) return num / (2.0f * p);
  return root_quot_slow(num, p);
}

__device__ __noinline__ float small_quot_slow(float num, float h) {
  return (float)((double)num / ((double)h + 0.00000001));
}

__device__ __noinline__ float small_quot(float num, float h) {
  const float c1 = 0x1.5798eep-27f;  // RN_f(1e-8)
  const float c2 = 0x1.18461cp-54f;  // RN_f(1e-8 - c1)
  // two-sum h + c1 = s + e exactly
  const float s = __fadd_rn(h, c1);
  const float bb = __fsub_rn(s, h);
  const float e = __fadd_rn(__fsub_rn(h, __fsub_rn(s, bb)), __fsub_rn(c1, bb));
  const float lo0 = __fadd_rn(e, c2);
  const float hi = __fadd_rn(s, lo0);
  const float lo = __fsub_rn(lo0, __fsub_rn(hi, s));
  // reject non-finite inputs, cancellation of h against 1e-8 (the pair then
  // misses the last bits of the double denominator), and tiny/huge values
  const float ah = fabsf(hi);
  if (!(ah > 1e-10f && ah < 1e30f) || !(fabsf(num) < 1e30f)) return small_quot_slow(num, h);
  const float q = __fdiv_rn(num, hi);
  const float aq = fabsf(q);
  if (q == 0.0f) {
    if (num == 0.0f) return q;  // signed zero of num / D
    return small_quot_slow(num, h);
  }
  if (!(aq > 1e-30f && aq < 1e30f)) return small_quot_slow(num, h);
  // N/D = q + (N - q*hi - q*lo)/(hi + lo); fma gives N - q*hi exactly
  const float r = __fmaf_rn(-q, hi, num);
  const float t = __fmaf_rn(-q, lo, r);
  const float corr = __fdiv_rn(t, hi);
  const float R = __fadd_rn(q, corr);
  // distance of the estimate from R, in units of R's half ulp
  const unsigned rb = __float_as_uint(R);
  if ((rb & 0x007fffffu) == 0u) return small_quot_slow(num, h);  // binade edge
  const float d = __fadd_rn(__fsub_rn(q, R), corr);              // ~ N/D - R
  const float half_ulp = __uint_as_float(((rb >> 23) & 0xffu) - 24u << 23);
  const float margin = __fmul_rn(fabsf(R), 0x1p-36f);
  if (fabsf(d) > half_ulp - margin) return small_quot_slow(num, h);
  return R;
}

// Tet update of apex D from A, B, C (metric Gram terms of the apex ordering).
__device__ __forceinline__ float tet_update(float TA, float TB, float TC, float ACAC, float ACBC,
                                            float ACCD, float BCBC, float BCCD, float CDCD) {
  if (TA >= kLarge3DDev && TB >= kLarge3DDev && TC >= kLarge3DDev) return kLarge3DDev;
  float p, q, r, l1, l2, l3, delta, TE;
  float fBC = kLarge3DDev, fAB = kLarge3DDev, fAC = kLarge3DDev, TD = kLarge3DDev;
  const float TAC = TC - TA;
  const float TBC = TC - TB;
  const float TAB = TB - TA;

  // ---- candidate on face BC (lambda1 = 0) ----
  p = BCBC * TBC * TBC - BCBC * BCBC;
  q = (BCCD + BCCD) * TBC * TBC - 2 * BCBC * BCCD;
  r = TBC * TBC * CDCD - BCCD * BCCD;
  delta = q * q - 4 * p * r;
  if (delta >= 0.0f) {
    l2 = root_quot(-q + sqrtf(delta), p);
    l3 = 1.0f - l2;
    if (l2 >= 0 && l2 <= 1) {
      TE = TB * l2 + TC * l3;
      fBC = fminf(fBC, TE + sqrtf((l2 * BCBC + BCCD) * l2 + (l2 * BCCD + CDCD)));
    }
    l2 = root_quot(-q - sqrtf(delta), p);
    l3 = 1.0f - l2;
    if (l2 >= 0 && l2 <= 1) {
      TE = TB * l2 + TC * l3;
      fBC = fminf(fBC, TE + sqrtf((l2 * BCBC + BCCD) * l2 + (l2 * BCCD + CDCD)));
    }
  }
  fBC = fminf(fBC, fminf(TB + sqrtf((BCBC + BCCD) + (BCCD + CDCD)), TC + sqrtf(CDCD)));

  // ---- candidate on face AB (lambda3 = 0) ----
  const float gx = ACAC - ACBC, gy = ACBC - BCBC, gz = ACCD - BCCD;
  p = (TAB * TAB * ACAC - gx * gx) + (BCBC * TAB * TAB - gy * gy) -
      ((ACBC + ACBC) * TAB * TAB - 2 * gx * gy);
  q = -(BCBC * TAB * TAB - gy * gy) * 2 + ((ACBC + ACBC) * TAB * TAB - 2 * gx * gy) +
      ((ACCD + ACCD) * TAB * TAB - 2 * gx * gz) - ((BCCD + BCCD) * TAB * TAB - 2 * gy * gz);
  r = (TAB * TAB * BCBC - gy * gy) + ((BCCD + BCCD) * TAB * TAB - 2 * gy * gz) +
      (TAB * TAB * CDCD - gz * gz);
  delta = q * q - 4 * p * r;
  if (delta >= 0.0f) {
    l1 = root_quot(-q + sqrtf(delta), p);
    l2 = 1 - l1;
    if (l1 >= 0 && l1 <= 1) {
      TE = TA * l1 + TB * l2;
      fAB = fminf(fAB, TE + sqrtf((l1 * ACAC + l2 * ACBC + ACCD) * l1 +
                                  (l1 * ACBC + l2 * BCBC + BCCD) * l2 +
                                  (l1 * ACCD + l2 * BCCD + CDCD)));
    }
    l1 = root_quot(-q - sqrtf(delta), p);
    l2 = 1 - l1;
    if (l1 >= 0 && l1 <= 1) {
      TE = TA * l1 + TB * l2;
      fAB = fminf(fAB, TE + sqrtf((l1 * ACAC + l2 * ACBC + ACCD) * l1 +
                                  (l1 * ACBC + l2 * BCBC + BCCD) * l2 +
                                  (l1 * ACCD + l2 * BCCD + CDCD)));
    }
  }
  fAB = fminf(fAB, fminf(TB + sqrtf((BCBC + BCCD) + (BCCD + CDCD)),
                         TA + sqrtf((ACAC + ACCD) + (ACCD + CDCD))));

  // ---- candidate on face AC (lambda2 = 0) ----
  p = ACAC * TAC * TAC - ACAC * ACAC;
  q = (ACCD + ACCD) * TAC * TAC - 2 * ACAC * ACCD;
  r = TAC * TAC * CDCD - ACCD * ACCD;
  delta = q * q - 4 * p * r;
  if (delta >= 0.0f) {
    l1 = root_quot(-q + sqrtf(delta), p);
    l3 = 1 - l1;
    if (l1 >= 0 && l1 <= 1) {
      TE = TA * l1 + TC * l3;
      fAC = fminf(fAC, TE + sqrtf((l1 * ACAC + ACCD) * l1 + (l1 * ACCD + CDCD)));
    }
    l1 = root_quot(-q - sqrtf(delta), p);
    l3 = 1 - l1;
    if (l1 >= 0 && l1 <= 1) {
      // the second candidate keeps a zero-weight TB term, as the reference does
      TE = TA * l1 + TB * 0.0f + TC * l3;
      fAC = fminf(fAC, TE + sqrtf((l1 * ACAC + ACCD) * l1 + (l1 * ACCD + CDCD)));
    }
  }
  fAC = fminf(fAC, fminf(TA + sqrtf((ACAC + ACCD) + (ACCD + CDCD)), TC + sqrtf(CDCD)));

  // ---- candidate inside face ABC: lambda2 = (s*lambda1 + t)/(h + 1e-8) ----
  const float s = TAC * ACBC - TBC * ACAC;
  const float t = TAC * BCCD - TBC * ACCD;
  const float h = -(TAC * BCBC - TBC * ACBC);
  p = (TAC * TAC * ACAC - ACAC * ACAC) * h * h + (BCBC * TAC * TAC - ACBC * ACBC) * s * s +
      ((ACBC + ACBC) * TAC * TAC - 2 * ACAC * ACBC) * s * h;
  q = (BCBC * TAC * TAC - ACBC * ACBC) * 2 * s * t +
      ((ACBC + ACBC) * TAC * TAC - 2 * ACAC * ACBC) * t * h +
      ((ACCD + ACCD) * TAC * TAC - 2 * ACAC * ACCD) * h * h +
      ((BCCD + BCCD) * TAC * TAC - 2 * ACBC * ACCD) * s * h;
  r = (TAC * TAC * BCBC - ACBC * ACBC) * t * t +
      ((BCCD + BCCD) * TAC * TAC - 2 * ACBC * ACCD) * t * h +
      (TAC * TAC * CDCD - ACCD * ACCD) * h * h;
  delta = q * q - 4 * p * r;
  if (delta >= 0.0f) {
    l1 = root_quot(-q + sqrtf(delta), p);
    l2 = small_quot(s * l1 + t, h);
    l3 = 1 - l1 - l2;
    if (l1 >= 0 && l1 <= 1 && l2 >= 0 && l2 <= 1 && l3 >= 0 && l3 <= 1) {
      TE = TA * l1 + TB * l2 + TC * l3;
      TD = fminf(TD, TE + sqrtf((l1 * ACAC + l2 * ACBC + ACCD) * l1 +
                                (l1 * ACBC + l2 * BCBC + BCCD) * l2 +
                                (l1 * ACCD + l2 * BCCD + CDCD)));
    }
    l1 = root_quot(-q - sqrtf(delta), p);
    l2 = small_quot(s * l1 + t, h);
    l3 = 1 - l1 - l2;
    if (l1 >= 0 && l1 <= 1 && l2 >= 0 && l2 <= 1 && l3 >= 0 && l3 <= 1) {
      TE = TA * l1 + TB * l2 + TC * l3;
      TD = fminf(TD, TE + sqrtf((l1 * ACAC + l2 * ACBC + ACCD) * l1 +
                                (l1 * ACBC + l2 * BCBC + BCCD) * l2 +
                                (l1 * ACCD + l2 * BCCD + CDCD)));
    }
  }
  TD = fminf(TD, fminf(fBC, fminf(fAB, fAC)));
  return TD;
}

// ---------------------------------------------------------------------------
// Explicitly rounded tet update.
//
// nvcc fuses a product into an adjacent sum (one FMA rounding instead of two), and
// in a sum or difference of two products it picks one of them; which one depends
// on the code around the expression, so the reference's four inlined updates in
// FIMCuda (CUDA_kernels.cu:454-457) do not all round alike, and the same source in
// a different kernel shape can round differently.  Here every product, sum,
// quotient and square root is one IEEE operation (__fmul_rn, __fadd_rn, __fmaf_rn,
// __fdiv_rn, __fsqrt_rn) that the compiler cannot fuse or split, so the result no
// longer depends on the surrounding code, and a mask states, for each sum or
// difference of two products (a site, numbered 0..51 in the order of the
// reference's statements), which product the reference's kernel fuses: bit S set =
// the second product is fused (x*y - z*w -> fma(-z, w, x*y)), clear = the first
// (fma(x, y, -(z*w))).
//
// The four masks below reproduce the reference kernel's own roundings for the four
// apex updates of a slot: they were fitted to, and reproduce bit for bit, the
// reference's FIMCuda run on 500,000 single-tet blocks (one sweep, so each vertex
// ends at that apex's update) covering jittered-cube tets with scalar metrics,
// slivers and random shapes with anisotropic metrics, and uniform random times;
// every site of the mask is exercised by those inputs (the one exception, site 29,
// is TB*0 beside TA*l1, where both choices give the same value).  A GPU test holds
// the group to the reference kernel on fresh inputs.
// ---------------------------------------------------------------------------
constexpr unsigned long long kFuseApexA = 0x6301902630000ull;  // update of A from B, D, C
constexpr unsigned long long kFuseApexB = 0x6301902630000ull;  // B from A, D, C
constexpr unsigned long long kFuseApexC = 0x4203182420002ull;  // C from A, B, D
constexpr unsigned long long kFuseApexD = 0x0000001100000000ull;  // D from A, B, C

// The masks agree at most sites; the others follow three flags of the apex kind:
// ab (A and B), abc (A, B and C), c (C alone).
struct ApexFuse {
  bool ab, abc, c;
};
constexpr unsigned long long fuse_mask(ApexFuse f) {
  const unsigned long long one = 1ull;
  return (one << 32 | one << 36) |
         (f.ab ? (one << 16 | one << 21 | one << 35 | one << 44 | one << 49) : 0ull) |
         (f.abc ? (one << 17 | one << 22 | one << 25 | one << 45 | one << 50) : 0ull) |
         (f.c ? (one << 1 | one << 31 | one << 37) : 0ull);
}
__host__ __device__ constexpr ApexFuse apex_fuse(int k) { return ApexFuse{k < 2, k < 3, k == 2}; }
static_assert(fuse_mask(apex_fuse(0)) == kFuseApexA && fuse_mask(apex_fuse(1)) == kFuseApexB &&
                  fuse_mask(apex_fuse(2)) == kFuseApexC && fuse_mask(apex_fuse(3)) == kFuseApexD,
              "the flags must give the fitted masks");

// x*y - z*w and x*y + z*w with the second (b) or the first product fused
__device__ __forceinline__ float x_ms(bool b, float x, float y, float z, float w) {
  const float pr = __fmul_rn(b ? x : z, b ? y : w);
  return __fmaf_rn(b ? -z : x, b ? w : y, b ? pr : -pr);
}
__device__ __forceinline__ float x_ma(bool b, float x, float y, float z, float w) {
  const float pr = __fmul_rn(b ? x : z, b ? y : w);
  return __fmaf_rn(b ? z : x, b ? w : y, pr);
}
// (l1*XX + l2*XY + XZ)*l1 + (l1*XY + l2*YY + YZ)*l2 + (l1*XZ + l2*YZ + ZZ): the metric
// length of the path from the apex to the point l1 A + l2 B + l3 C
__device__ __forceinline__ float x_dist3(ApexFuse f, float l1, float l2, float ACAC, float ACBC, float ACCD,
                                         float BCBC, float BCCD, float CDCD) {
  const float X = __fadd_rn(__fmaf_rn(l1, ACAC, __fmul_rn(l2, ACBC)), ACCD);
  const float Y = __fadd_rn(x_ma(f.ab, l1, ACBC, l2, BCBC), BCCD);
  const float Z = __fadd_rn(x_ma(f.abc, l1, ACCD, l2, BCCD), CDCD);
  return __fadd_rn(__fmaf_rn(X, l1, __fmul_rn(Y, l2)), Z);
}
// (l*XX + XY)*l + (l*XY + YY): the same on an edge
__device__ __forceinline__ float x_dist2(float l, float XX, float XY, float YY) {
  return __fmaf_rn(__fmaf_rn(l, XX, XY), l, __fmaf_rn(l, XY, YY));
}
__device__ __forceinline__ float x_root(float num, float p) {
  if (fabsf(p) < 0x1p126f) return __fdiv_rn(num, __fmul_rn(2.0f, p));
  return root_quot_slow(num, p);
}

// localSolverTet1 (CUDA_kernels.cu:69-225) takes the least of the candidates on the
// face's edges BC, AB and AC and inside the face ABC.  A minimum does not depend on its
// order (a NaN candidate is ignored wherever it stands), so the update is written as one
// function per edge and one for the inside, each starting from LARGENUM as the
// reference's candidates do.

// Edge XC, X = B or A: sites 0-5 (BC) and 24-29 (AC).  AC's second candidate keeps a
// zero-weight TB term in the reference, which leaves TA*l1 rounded by itself; its sum
// is then the one with the second product fused.
__device__ __forceinline__ float tet_part_edge(bool ac, ApexFuse f, float TX, float TC, float XX, float XC, float CC) {
  const float T = __fsub_rn(TC, TX);
  const float p = __fmaf_rn(__fmul_rn(XX, T), T, -__fmul_rn(XX, XX));
  const float q = x_ms(ac ? f.abc : f.c, __fmul_rn(__fadd_rn(XC, XC), T), T, __fmul_rn(2.0f, XX), XC);
  const float r = __fmaf_rn(__fmul_rn(T, T), CC, -__fmul_rn(XC, XC));
  const float delta = __fmaf_rn(q, q, -__fmul_rn(__fmul_rn(4.0f, p), r));
  float best = fminf(__fadd_rn(TX, __fsqrt_rn(__fadd_rn(__fadd_rn(XX, XC), __fadd_rn(XC, CC)))),
                     __fadd_rn(TC, __fsqrt_rn(CC)));
  best = fminf(kLarge3DDev, best);
  if (delta >= 0.0f) {
    const float sd = __fsqrt_rn(delta);
    float l = x_root(__fadd_rn(-q, sd), p);
    float m = __fsub_rn(1.0f, l);
    if (l >= 0 && l <= 1)
      best = fminf(best, __fadd_rn(__fmaf_rn(TX, l, __fmul_rn(TC, m)), __fsqrt_rn(x_dist2(l, XX, XC, CC))));
    l = x_root(__fsub_rn(-q, sd), p);
    m = __fsub_rn(1.0f, l);
    if (l >= 0 && l <= 1)
      best = fminf(best, __fadd_rn(x_ma(ac, TX, l, TC, m), __fsqrt_rn(x_dist2(l, XX, XC, CC))));
  }
  return best;
}
// Edge AB (sites 6-23); its end points are candidates of the other two edges.
__device__ __forceinline__ float tet_part_ab(ApexFuse f, float TA, float TB, float ACAC, float ACBC, float ACCD,
                                             float BCBC, float BCCD, float CDCD) {
  const float TAB = __fsub_rn(TB, TA);
  const float gx = __fsub_rn(ACAC, ACBC), gy = __fsub_rn(ACBC, BCBC), gz = __fsub_rn(ACCD, BCCD);
  const float TAB2 = __fmul_rn(TAB, TAB);
  const float P1 = __fmaf_rn(TAB2, ACAC, -__fmul_rn(gx, gx));
  const float P2 = __fmaf_rn(__fmul_rn(BCBC, TAB), TAB, -__fmul_rn(gy, gy));
  const float P3 = __fmaf_rn(__fmul_rn(__fadd_rn(ACBC, ACBC), TAB), TAB, -__fmul_rn(__fmul_rn(2.0f, gx), gy));
  const float p = __fsub_rn(__fadd_rn(P1, P2), P3);
  const float P4 = __fmaf_rn(__fmul_rn(__fadd_rn(ACCD, ACCD), TAB), TAB, -__fmul_rn(__fmul_rn(2.0f, gx), gz));
  const float P5 = __fmaf_rn(__fmul_rn(__fadd_rn(BCCD, BCCD), TAB), TAB, -__fmul_rn(__fmul_rn(2.0f, gy), gz));
  const float q = __fsub_rn(__fadd_rn(__fadd_rn(__fmul_rn(-P2, 2.0f), P3), P4), P5);
  const float r = __fadd_rn(__fadd_rn(__fmaf_rn(TAB2, BCBC, -__fmul_rn(gy, gy)), P5),
                            __fmaf_rn(TAB2, CDCD, -__fmul_rn(gz, gz)));
  const float delta = __fmaf_rn(q, q, -__fmul_rn(__fmul_rn(4.0f, p), r));
  float best = kLarge3DDev;
  if (delta >= 0.0f) {
    const float sd = __fsqrt_rn(delta);
    float l1 = x_root(__fadd_rn(-q, sd), p);
    float l2 = __fsub_rn(1.0f, l1);
    if (l1 >= 0 && l1 <= 1)
      best = fminf(best, __fadd_rn(__fmaf_rn(TA, l1, __fmul_rn(TB, l2)),
                                   __fsqrt_rn(x_dist3(f, l1, l2, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD))));
    l1 = x_root(__fsub_rn(-q, sd), p);
    l2 = __fsub_rn(1.0f, l1);
    if (l1 >= 0 && l1 <= 1)
      best = fminf(best, __fadd_rn(__fmaf_rn(TA, l1, __fmul_rn(TB, l2)),
                                   __fsqrt_rn(x_dist3(f, l1, l2, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD))));
  }
  return best;
}
// Inside the face ABC, lambda2 = (s*lambda1 + t)/(h + 1e-8) (sites 30-51): the
// candidate of the quadratic's root with +sqrt (minus = false) or -sqrt.
struct TetInner {
  float p, q, s, t, h, sd;  // sd < 0: no real root
};
__device__ __forceinline__ TetInner tet_inner_setup(ApexFuse f, float TA, float TB, float TC, float ACAC, float ACBC,
                                                    float ACCD, float BCBC, float BCCD, float CDCD) {
  TetInner o;
  const float TAC = __fsub_rn(TC, TA), TBC = __fsub_rn(TC, TB);
  const float TAC2 = __fmul_rn(TAC, TAC);
  const float qAC = x_ms(f.abc, __fmul_rn(__fadd_rn(ACCD, ACCD), TAC), TAC, __fmul_rn(2.0f, ACAC), ACCD);
  const float rAC = __fmaf_rn(TAC2, CDCD, -__fmul_rn(ACCD, ACCD));
  const float s = __fmaf_rn(TAC, ACBC, -__fmul_rn(TBC, ACAC));
  const float t = x_ms(f.c, TAC, BCCD, TBC, ACCD);
  const float h = -__fmaf_rn(-TBC, ACBC, __fmul_rn(TAC, BCBC));
  const float A1 = __fmaf_rn(TAC2, ACAC, -__fmul_rn(ACAC, ACAC));
  const float A2 = __fmaf_rn(__fmul_rn(BCBC, TAC), TAC, -__fmul_rn(ACBC, ACBC));
  const float A3 = x_ms(f.ab, __fmul_rn(__fadd_rn(ACBC, ACBC), TAC), TAC, __fmul_rn(2.0f, ACAC), ACBC);
  const float A4 = x_ms(f.c, __fmul_rn(__fadd_rn(BCCD, BCCD), TAC), TAC, __fmul_rn(2.0f, ACBC), ACCD);
  o.p = __fmaf_rn(__fmul_rn(A3, s), h, __fmaf_rn(__fmul_rn(A2, s), s, __fmul_rn(__fmul_rn(A1, h), h)));
  o.q = __fmaf_rn(__fmul_rn(A4, s), h,
                  __fmaf_rn(__fmul_rn(qAC, h), h,
                            __fmaf_rn(__fmul_rn(__fmul_rn(A2, 2.0f), s), t, __fmul_rn(__fmul_rn(A3, t), h))));
  const float r = __fmaf_rn(__fmul_rn(rAC, h), h,
                            __fmaf_rn(__fmul_rn(__fmaf_rn(TAC2, BCBC, -__fmul_rn(ACBC, ACBC)), t), t,
                                      __fmul_rn(__fmul_rn(A4, t), h)));
  const float delta = __fmaf_rn(o.q, o.q, -__fmul_rn(__fmul_rn(4.0f, o.p), r));
  o.s = s;
  o.t = t;
  o.h = h;
  o.sd = (delta >= 0.0f) ? __fsqrt_rn(delta) : -1.0f;
  return o;
}
__device__ __forceinline__ float tet_inner_root(const TetInner& o, bool minus, ApexFuse f, float TA, float TB, float TC,
                                                float ACAC, float ACBC, float ACCD, float BCBC, float BCCD,
                                                float CDCD) {
  const float l1 = x_root(__fadd_rn(-o.q, minus ? -o.sd : o.sd), o.p);
  if (!(l1 >= 0 && l1 <= 1)) return kLarge3DDev;
  const float l2 = small_quot(__fmaf_rn(o.s, l1, o.t), o.h);
  const float l3 = __fsub_rn(__fsub_rn(1.0f, l1), l2);
  if (!(l2 >= 0 && l2 <= 1 && l3 >= 0 && l3 <= 1)) return kLarge3DDev;
  return fminf(kLarge3DDev, __fadd_rn(__fmaf_rn(TC, l3, __fmaf_rn(TA, l1, __fmul_rn(TB, l2))),
                                      __fsqrt_rn(x_dist3(f, l1, l2, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD))));
}
// The update of apex k's argument order, or its least candidate among `parts` (uniform
// across a warp: bits 0 edge BC, 1 edge AC, 2 edge AB, 3 and 4 the inner roots with
// +sqrt and -sqrt); out of line, one body for all apex kinds, which spares the
// instruction cache and lets a warp's lanes update different apexes.
constexpr unsigned kAllParts = 31u;
__device__ __noinline__ float tet_update_parts(unsigned parts, int k, float TA, float TB, float TC, float ACAC,
                                               float ACBC, float ACCD, float BCBC, float BCCD, float CDCD) {
  if (TA >= kLarge3DDev && TB >= kLarge3DDev && TC >= kLarge3DDev) return kLarge3DDev;
  const ApexFuse f = apex_fuse(k);
  float best = kLarge3DDev;
  if (parts & 1u) best = tet_part_edge(false, f, TB, TC, BCBC, BCCD, CDCD);
  if (parts & 2u) best = fminf(best, tet_part_edge(true, f, TA, TC, ACAC, ACCD, CDCD));
  if (parts & 4u) best = fminf(best, tet_part_ab(f, TA, TB, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD));
  if (parts & 24u) {
    const TetInner o = tet_inner_setup(f, TA, TB, TC, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD);
    if (o.sd >= 0.0f) {
      if (parts & 8u) best = fminf(best, tet_inner_root(o, false, f, TA, TB, TC, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD));
      if (parts & 16u) best = fminf(best, tet_inner_root(o, true, f, TA, TB, TC, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD));
    }
  }
  return best;
}

// The remaining metric edge products of a slot from its six stored ones
// (CUDA_kernels.cu:429-437), in the order the tet updates take them.
struct TetGram {
  float ACAC, ACBC, ACCD, BCBC, BCCD, CDCD, ADAD, ADBD, ADCD, BDBD, CDBD;
};
__device__ __forceinline__ TetGram tet_gram9(float ACBC, float BCCD, float ACCD, float ADBD, float ACAD, float BCBD) {
  TetGram g;
  const float ADBC = __fadd_rn(ACBC, BCCD);
  const float ACBD = __fadd_rn(ACBC, ACCD);
  g.CDBD = __fsub_rn(ADBD, ACBD);
  g.ADCD = __fsub_rn(ADBD, ADBC);
  g.CDCD = __fsub_rn(g.ADCD, ACCD);
  g.ADAD = __fadd_rn(g.ADCD, ACAD);
  g.ACAC = __fsub_rn(ACAD, ACCD);
  g.BDBD = __fadd_rn(BCBD, g.CDBD);
  g.BCBC = __fsub_rn(BCBD, BCCD);
  g.ACBC = ACBC;
  g.BCCD = BCCD;
  g.ACCD = ACCD;
  g.ADBD = ADBD;
  return g;
}

// An apex update's arguments: the times of its face's corners and the metric products
// as the reference passes them for apex k (0..3 = A, B, C, D).  k may differ between the
// lanes of a warp: every argument is picked by selects.
__device__ __forceinline__ float apex_update(int k, const float T[4], const TetGram& g, unsigned parts = kAllParts) {
  const bool a = k == 0, c = k == 2, ab = k < 2;
  return tet_update_parts(parts, k, a ? T[1] : T[0], ab ? T[3] : T[1], c ? T[3] : T[2], a ? g.BCBC : c ? g.ADAD : g.ACAC,
                          a ? -g.BCCD : c ? g.ADBD : ab ? -g.ACCD : g.ACBC, ab ? -g.ACBC : c ? -g.ADCD : g.ACCD,
                          ab ? g.CDCD : c ? g.BDBD : g.BCBC, a ? g.ACCD : c ? -g.CDBD : g.BCCD,
                          a ? g.ACAC : ab ? g.BCBC : g.CDCD);
}

// The operations of the wide (precision mode) update, named so the update reads
// like the FP32 one.
__device__ __forceinline__ double w_make(double a, double) { return a; }
__device__ __forceinline__ double w_min(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ double w_sqrt(double a) { return sqrt(a); }
__device__ __forceinline__ double w_recip(double a) { return 1.0 / a; }
__device__ __forceinline__ bool w_ge0(double a) { return a >= 0.0; }
__device__ __forceinline__ bool w_in01(double a) { return a >= 0 && a <= 1; }
__device__ __forceinline__ bool w_large(double a) { return a >= (double)kLarge3DDev; }
__device__ __forceinline__ float w_float(double a) { return (float)a; }

// Square root of a non-negative candidate distance for the FP64 update: the
// argument is formed in FP64 (where the cancellation is), the root taken in FP32 (relative error below 1e-7, far inside the scheme's 1e-5 tolerance), which
// spares the slow FP64 unit.
__device__ __forceinline__ double sqrt_pos(double x) { return (double)sqrtf((float)x); }

// The same tet update carried out in FP64 (precision mode: slots of sliver or
// ill-conditioned tets), written over a type R for the helpers above.  Same
// candidates and order as tet_update; the metric edge products come from FP64 setup
// values, quotients are FP64 (one reciprocal per candidate face); only the candidate
// roots use sqrt_pos.  (A double-float R, two FP32 numbers per value, ran slower on
// GB300 than the FP64 unit and was dropped.)
template <typename R>
__device__ __forceinline__ R tet_update_wide(R TA, R TB, R TC, R ACAC, R ACBC, R ACCD, R BCBC, R BCCD, R CDCD) {
  const R L = w_make((double)kLarge3DDev, R{});
  if (w_large(TA) && w_large(TB) && w_large(TC)) return L;
  const R one = w_make(1.0, R{}), eps8 = w_make(0.00000001, R{});
  R p, q, r, l1, l2, l3, delta, TE;
  R fBC = L, fAB = L, fAC = L, TD = L;
  const R TAC = TC - TA, TBC = TC - TB, TAB = TB - TA;
  // face BC
  p = BCBC * TBC * TBC - BCBC * BCBC;
  q = (BCCD + BCCD) * TBC * TBC - 2.0f * BCBC * BCCD;
  r = TBC * TBC * CDCD - BCCD * BCCD;
  delta = q * q - 4.0f * p * r;
  if (w_ge0(delta)) {
    const R sd = w_sqrt(delta), i2p = w_recip(2.0f * p);
    for (int sg = 0; sg < 2; ++sg) {
      l2 = (-q + (sg ? -sd : sd)) * i2p;
      l3 = one - l2;
      if (w_in01(l2)) {
        TE = TB * l2 + TC * l3;
        fBC = w_min(fBC, TE + sqrt_pos((l2 * BCBC + BCCD) * l2 + (l2 * BCCD + CDCD)));
      }
    }
  }
  fBC = w_min(fBC, w_min(TB + sqrt_pos((BCBC + BCCD) + (BCCD + CDCD)), TC + sqrt_pos(CDCD)));
  // face AB
  const R gx = ACAC - ACBC, gy = ACBC - BCBC, gz = ACCD - BCCD;
  p = (TAB * TAB * ACAC - gx * gx) + (BCBC * TAB * TAB - gy * gy) - ((ACBC + ACBC) * TAB * TAB - 2.0f * gx * gy);
  q = -(BCBC * TAB * TAB - gy * gy) * w_make(2.0, R{}) + ((ACBC + ACBC) * TAB * TAB - 2.0f * gx * gy) +
      ((ACCD + ACCD) * TAB * TAB - 2.0f * gx * gz) - ((BCCD + BCCD) * TAB * TAB - 2.0f * gy * gz);
  r = (TAB * TAB * BCBC - gy * gy) + ((BCCD + BCCD) * TAB * TAB - 2.0f * gy * gz) + (TAB * TAB * CDCD - gz * gz);
  delta = q * q - 4.0f * p * r;
  if (w_ge0(delta)) {
    const R sd = w_sqrt(delta), i2p = w_recip(2.0f * p);
    for (int sg = 0; sg < 2; ++sg) {
      l1 = (-q + (sg ? -sd : sd)) * i2p;
      l2 = one - l1;
      if (w_in01(l1)) {
        TE = TA * l1 + TB * l2;
        fAB = w_min(fAB, TE + sqrt_pos((l1 * ACAC + l2 * ACBC + ACCD) * l1 + (l1 * ACBC + l2 * BCBC + BCCD) * l2 +
                                       (l1 * ACCD + l2 * BCCD + CDCD)));
      }
    }
  }
  fAB = w_min(fAB, w_min(TB + sqrt_pos((BCBC + BCCD) + (BCCD + CDCD)), TA + sqrt_pos((ACAC + ACCD) + (ACCD + CDCD))));
  // face AC
  p = ACAC * TAC * TAC - ACAC * ACAC;
  q = (ACCD + ACCD) * TAC * TAC - 2.0f * ACAC * ACCD;
  r = TAC * TAC * CDCD - ACCD * ACCD;
  delta = q * q - 4.0f * p * r;
  if (w_ge0(delta)) {
    const R sd = w_sqrt(delta), i2p = w_recip(2.0f * p);
    for (int sg = 0; sg < 2; ++sg) {
      l1 = (-q + (sg ? -sd : sd)) * i2p;
      l3 = one - l1;
      if (w_in01(l1)) {
        TE = TA * l1 + TC * l3;
        fAC = w_min(fAC, TE + sqrt_pos((l1 * ACAC + ACCD) * l1 + (l1 * ACCD + CDCD)));
      }
    }
  }
  fAC = w_min(fAC, w_min(TA + sqrt_pos((ACAC + ACCD) + (ACCD + CDCD)), TC + sqrt_pos(CDCD)));
  // inside face ABC
  const R s = TAC * ACBC - TBC * ACAC;
  const R t = TAC * BCCD - TBC * ACCD;
  const R h = -(TAC * BCBC - TBC * ACBC);
  p = (TAC * TAC * ACAC - ACAC * ACAC) * h * h + (BCBC * TAC * TAC - ACBC * ACBC) * s * s +
      ((ACBC + ACBC) * TAC * TAC - 2.0f * ACAC * ACBC) * s * h;
  q = (BCBC * TAC * TAC - ACBC * ACBC) * w_make(2.0, R{}) * s * t +
      ((ACBC + ACBC) * TAC * TAC - 2.0f * ACAC * ACBC) * t * h +
      ((ACCD + ACCD) * TAC * TAC - 2.0f * ACAC * ACCD) * h * h +
      ((BCCD + BCCD) * TAC * TAC - 2.0f * ACBC * ACCD) * s * h;
  r = (TAC * TAC * BCBC - ACBC * ACBC) * t * t + ((BCCD + BCCD) * TAC * TAC - 2.0f * ACBC * ACCD) * t * h +
      (TAC * TAC * CDCD - ACCD * ACCD) * h * h;
  delta = q * q - 4.0f * p * r;
  if (w_ge0(delta)) {
    const R sd = w_sqrt(delta), i2p = w_recip(2.0f * p), ih = w_recip(h + eps8);
    for (int sg = 0; sg < 2; ++sg) {
      l1 = (-q + (sg ? -sd : sd)) * i2p;
      l2 = (s * l1 + t) * ih;
      l3 = one - l1 - l2;
      if (w_in01(l1) && w_in01(l2) && w_in01(l3)) {
        TE = TA * l1 + TB * l2 + TC * l3;
        TD = w_min(TD, TE + sqrt_pos((l1 * ACAC + l2 * ACBC + ACCD) * l1 + (l1 * ACBC + l2 * BCBC + BCCD) * l2 +
                                     (l1 * ACCD + l2 * BCCD + CDCD)));
      }
    }
  }
  return w_min(TD, w_min(fBC, w_min(fAB, fAC)));
}
__device__ __forceinline__ double tet_update_f64(double TA, double TB, double TC, double ACAC, double ACBC,
                                                 double ACCD, double BCBC, double BCCD, double CDCD) {
  return tet_update_wide<double>(TA, TB, TC, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD);
}

// The same update of apex k with its roundings written out: each fused multiply-add is
// the one the compiler chose for tet_update_wide in the kernel that ran precision mode
// before, so the results do not depend on the code around it.  The choice matters where
// two corners' times nearly agree: p, q and r then cancel, and a discriminant's sign
// decides whether a slab of the face counts at all.  One rule covers the four kinds (the
// products of t and of BCCD's row are fused the other way round for A, B, C and for C);
// it reproduces that kernel's bits on 512 000 updates, two thirds of them with two times
// within 600 units in the last place.  One body for all kinds: the lanes of a warp
// update different apexes.  `parts` as in tet_update_parts.
__device__ __forceinline__ double d_ms(bool b, double x, double y, double z, double w) {  // x*y - z*w
  const double pr = __dmul_rn(b ? x : z, b ? y : w);
  return __fma_rn(b ? -z : x, b ? w : y, b ? pr : -pr);
}
__device__ __forceinline__ double d_root(double q, double sd, double i2p) { return __dmul_rn(__dadd_rn(-q, sd), i2p); }
__device__ __forceinline__ double d_dist3(double l1, double l2, double ACAC, double ACBC, double ACCD, double BCBC,
                                          double BCCD, double CDCD) {
  const double X = __fma_rn(l1, ACAC, __fma_rn(l2, ACBC, ACCD)), Y = __fma_rn(l1, ACBC, __fma_rn(l2, BCBC, BCCD));
  return __fma_rn(X, l1, __fma_rn(Y, l2, __fma_rn(l1, ACCD, __fma_rn(l2, BCCD, CDCD))));
}
// an edge XC of the face: its inner candidates and its end points
__device__ __forceinline__ double tet64_part_edge(double TX, double TC, double XX, double XC, double CC) {
  const double T = __dsub_rn(TC, TX), XC2 = __dadd_rn(XC, XC);
  const double p = d_ms(false, __dmul_rn(XX, T), T, XX, XX);
  const double q = d_ms(false, __dmul_rn(XC2, T), T, __dmul_rn(2.0, XX), XC);
  const double r = d_ms(false, __dmul_rn(T, T), CC, XC, XC);
  const double delta = d_ms(false, q, q, __dmul_rn(4.0, p), r);
  double best = fmin(__dadd_rn(TX, sqrt_pos(__dadd_rn(__dadd_rn(XX, XC), __dadd_rn(XC, CC)))), __dadd_rn(TC, sqrt_pos(CC)));
  best = fmin((double)kLarge3DDev, best);
  if (delta >= 0.0) {
    const double sd = __dsqrt_rn(delta), i2p = __drcp_rn(__dmul_rn(2.0, p));
#pragma unroll 1
    for (int sg = 0; sg < 2; ++sg) {
      const double l = d_root(q, sg ? -sd : sd, i2p), m = __dsub_rn(1.0, l);
      if (l >= 0 && l <= 1)
        best = fmin(best, __dadd_rn(__fma_rn(TX, l, __dmul_rn(TC, m)),
                                    sqrt_pos(__fma_rn(__fma_rn(l, XX, XC), l, __fma_rn(l, XC, CC)))));
    }
  }
  return best;
}
// edge AB; its end points are candidates of the other two edges
__device__ __forceinline__ double tet64_part_ab(double TA, double TB, double ACAC, double ACBC, double ACCD, double BCBC,
                                                double BCCD, double CDCD) {
  const double T = __dsub_rn(TB, TA), T2 = __dmul_rn(T, T);
  const double gx = __dsub_rn(ACAC, ACBC), gy = __dsub_rn(ACBC, BCBC), gz = __dsub_rn(ACCD, BCCD);
  const double P1 = d_ms(false, T2, ACAC, gx, gx), P2 = d_ms(false, __dmul_rn(BCBC, T), T, gy, gy);
  const double P3 = d_ms(false, __dmul_rn(__dadd_rn(ACBC, ACBC), T), T, __dmul_rn(2.0, gx), gy);
  const double P4 = d_ms(false, __dmul_rn(__dadd_rn(ACCD, ACCD), T), T, __dmul_rn(2.0, gx), gz);
  const double P5 = d_ms(false, __dmul_rn(__dadd_rn(BCCD, BCCD), T), T, __dmul_rn(2.0, gy), gz);
  const double p = __dsub_rn(__dadd_rn(P1, P2), P3);
  const double q = __dsub_rn(__dadd_rn(__dadd_rn(__dmul_rn(-P2, 2.0), P3), P4), P5);
  const double r = __dadd_rn(__dadd_rn(d_ms(false, T2, BCBC, gy, gy), P5), d_ms(false, T2, CDCD, gz, gz));
  const double delta = d_ms(false, q, q, __dmul_rn(4.0, p), r);
  double best = (double)kLarge3DDev;
  if (delta >= 0.0) {
    const double sd = __dsqrt_rn(delta), i2p = __drcp_rn(__dmul_rn(2.0, p));
#pragma unroll 1
    for (int sg = 0; sg < 2; ++sg) {
      const double l1 = d_root(q, sg ? -sd : sd, i2p), l2 = __dsub_rn(1.0, l1);
      if (l1 >= 0 && l1 <= 1) {
        const double X = __dadd_rn(__fma_rn(l1, ACAC, __dmul_rn(l2, ACBC)), ACCD);
        const double Y = __dadd_rn(__fma_rn(l1, ACBC, __dmul_rn(l2, BCBC)), BCCD);
        const double Z = __dadd_rn(__fma_rn(l1, ACCD, __dmul_rn(l2, BCCD)), CDCD);
        best = fmin(best, __dadd_rn(__fma_rn(TA, l1, __dmul_rn(TB, l2)),
                                    sqrt_pos(__dadd_rn(__dadd_rn(__dmul_rn(X, l1), __dmul_rn(Y, l2)), Z))));
      }
    }
  }
  return best;
}
// inside the face: roots with +sqrt (parts bit 3) and -sqrt (bit 4)
__device__ __forceinline__ double tet64_part_inner(unsigned parts, int k, double TA, double TB, double TC, double ACAC,
                                                   double ACBC, double ACCD, double BCBC, double BCCD, double CDCD) {
  const double TAC = __dsub_rn(TC, TA), TBC = __dsub_rn(TC, TB), TAC2 = __dmul_rn(TAC, TAC);
  const double s = d_ms(false, TAC, ACBC, TBC, ACAC);
  const double t = d_ms(k < 3, TAC, BCCD, TBC, ACCD);
  const double h = -d_ms(true, TAC, BCBC, TBC, ACBC);
  const double P1 = d_ms(false, TAC2, ACAC, ACAC, ACAC), P2 = d_ms(false, __dmul_rn(BCBC, TAC), TAC, ACBC, ACBC);
  const double P3 = d_ms(false, __dmul_rn(__dadd_rn(ACBC, ACBC), TAC), TAC, __dmul_rn(2.0, ACAC), ACBC);
  const double P4 = d_ms(false, __dmul_rn(__dadd_rn(ACCD, ACCD), TAC), TAC, __dmul_rn(2.0, ACAC), ACCD);
  const double P5 = d_ms(k == 2, __dmul_rn(__dadd_rn(BCCD, BCCD), TAC), TAC, __dmul_rn(2.0, ACBC), ACCD);
  const double P6 = d_ms(false, TAC2, BCBC, ACBC, ACBC), P7 = d_ms(false, TAC2, CDCD, ACCD, ACCD);
  const double p = __fma_rn(__dmul_rn(P3, s), h, __fma_rn(__dmul_rn(P2, s), s, __dmul_rn(__dmul_rn(P1, h), h)));
  double q = __fma_rn(__dmul_rn(__dmul_rn(P2, 2.0), s), t, __dmul_rn(__dmul_rn(P3, t), h));
  q = __fma_rn(__dmul_rn(P5, s), h, __fma_rn(__dmul_rn(P4, h), h, q));
  const double r =
      __fma_rn(__dmul_rn(P7, h), h, __fma_rn(__dmul_rn(P6, t), t, __dmul_rn(__dmul_rn(P5, t), h)));
  const double delta = d_ms(false, q, q, __dmul_rn(4.0, p), r);
  double best = (double)kLarge3DDev;
  if (delta >= 0.0) {
    const double sd = __dsqrt_rn(delta), i2p = __drcp_rn(__dmul_rn(2.0, p)), ih = __drcp_rn(__dadd_rn(h, 0.00000001));
#pragma unroll 1
    for (int sg = 0; sg < 2; ++sg) {
      if (!((parts >> (3 + sg)) & 1u)) continue;
      const double l1 = d_root(q, sg ? -sd : sd, i2p), l2 = __dmul_rn(__fma_rn(s, l1, t), ih);
      const double l3 = __dsub_rn(__dsub_rn(1.0, l1), l2);
      if (l1 >= 0 && l1 <= 1 && l2 >= 0 && l2 <= 1 && l3 >= 0 && l3 <= 1)
        best = fmin(best, __dadd_rn(__fma_rn(TC, l3, __fma_rn(TA, l1, __dmul_rn(TB, l2))),
                                    sqrt_pos(d_dist3(l1, l2, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD))));
    }
  }
  return best;
}
__device__ __noinline__ float tet64_update_parts(unsigned parts, int k, double TA, double TB, double TC, double ACAC,
                                                 double ACBC, double ACCD, double BCBC, double BCCD, double CDCD) {
  const double L = (double)kLarge3DDev;
  if (TA >= L && TB >= L && TC >= L) return kLarge3DDev;
  double best = L;
  if (parts & 1u) best = tet64_part_edge(TB, TC, BCBC, BCCD, CDCD);
  if (parts & 2u) best = fmin(best, tet64_part_edge(TA, TC, ACAC, ACCD, CDCD));
  if (parts & 4u) best = fmin(best, tet64_part_ab(TA, TB, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD));
  if (parts & 24u) best = fmin(best, tet64_part_inner(parts, k, TA, TB, TC, ACAC, ACBC, ACCD, BCBC, BCCD, CDCD));
  return (float)best;
}
// Apex k of a slot with corner times T and the six products g, as apex_update.
__device__ __forceinline__ float apex_update64(int k, const float T[4], const double g[6], unsigned parts = kAllParts) {
  const double ACBC = g[0], BCCD = g[1], ACCD = g[2], ADBD = g[3], ACAD = g[4], BCBD = g[5];
  const double ADBC = __dadd_rn(ACBC, BCCD), ACBD = __dadd_rn(ACBC, ACCD);
  const double CDBD = __dsub_rn(ADBD, ACBD), ADCD = __dsub_rn(ADBD, ADBC);
  const double CDCD = __dsub_rn(ADCD, ACCD), ADAD = __dadd_rn(ADCD, ACAD), ACAC = __dsub_rn(ACAD, ACCD);
  const double BDBD = __dadd_rn(BCBD, CDBD), BCBC = __dsub_rn(BCBD, BCCD);
  const bool a = k == 0, c = k == 2, ab = k < 2;
  return tet64_update_parts(parts, k, a ? T[1] : T[0], ab ? T[3] : T[1], c ? T[3] : T[2], a ? BCBC : c ? ADAD : ACAC,
                            a ? -BCCD : c ? ADBD : ab ? -ACCD : ACBC, ab ? -ACBC : c ? -ADCD : ACCD,
                            ab ? CDCD : c ? BDBD : BCBC, a ? ACCD : c ? -CDBD : BCCD, a ? ACAC : ab ? BCBC : CDCD);
}

// Triangle update of corner C from A and B; F is the inverse speed.  Uses the
// reference's MIN macro semantics ((a)<(b)?(a):(b)), not fminf.
__device__ __forceinline__ float mn2(float a, float b) { return (a < b) ? a : b; }

//
// kHoisted: inside the reference's multi-sweep FIMCuda the products LenAC*F and
// LenBC*F do not change between sweeps and are rounded once before the sweeps,
// so the edge candidates there are TA + RN(LenAC*F); the single-sweep check
// kernel fuses them into one multiply-add.  EA, EB carry the pre-rounded products
// in the first form and are ignored in the second.
template <bool kHoisted>
__device__ __forceinline__ float tri_update(float TA, float TB, float TC, float LenAB, float LenBC,
                                            float LenAC, float F, float EA, float EB) {
  float TC1 = kLarge2DDev, TC2 = kLarge2DDev;
  const float TAB = TB - TA;
  const float a = (F * F * LenAB * LenAB - TAB * TAB) * LenAB * LenAB;
  const float EdgeTA = kHoisted ? TA + EA : TA + LenAC * F;
  const float EdgeTB = kHoisted ? TB + EB : TB + LenBC * F;
  if (a > 0.0f) {
    const float cosA = (LenAC * LenAC + LenAB * LenAB - LenBC * LenBC) / (2.0f * LenAC * LenAB);
    const float b = 2.0f * LenAB * LenAC * cosA * (TAB * TAB - F * F * LenAB * LenAB);
    const float delta = 4.0f * LenAC * LenAC * a * TAB * TAB * (1.0f - cosA * cosA);
    const float l1 = (-b + sqrtf(delta)) / (2.0f * a);
    const float l2 = (-b - sqrtf(delta)) / (2.0f * a);
    if (l1 >= 0.0f && l1 <= 1.0f) {
      const float LenAD = l1 * LenAB;
      const float LenCD = sqrtf(LenAC * LenAC + LenAD * LenAD - 2 * LenAC * LenAD * cosA);
      TC1 = l1 * TAB + TA + LenCD * F;
    }
    if (l2 >= 0.0f && l2 <= 1.0f) {
      const float LenAD = l2 * LenAB;
      const float LenCD = sqrtf(LenAC * LenAC + LenAD * LenAD - 2 * LenAC * LenAD * cosA);
      TC2 = l2 * TAB + TA + LenCD * F;
    }
    return mn2(TC, mn2(TC2, mn2(TC1, mn2(EdgeTA, EdgeTB))));
  }
  return mn2(TC, mn2(EdgeTA, EdgeTB));
}

}  // namespace eikgb
