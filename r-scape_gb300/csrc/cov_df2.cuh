// cov_df2.cuh -- double-float arithmetic on two values at once, with the
// packed FP32 instructions of sm_100 and later (add/mul/fma.rn.f32x2: one
// instruction, two independent IEEE results).
//
// A packed instruction holds the FMA pipe for two cycles, so it does not raise
// the pipe's peak; it halves the issue slots and the instruction bytes of a
// long unrolled body, and puts two independent chains behind every
// dependency.  Each half rounds exactly as the scalar operation of
// cov_df.cuh.  The instructions take no negated operand, so the
// transformations below are written with subtractions, and products that are
// only subtracted are formed negated (-p = (-a) b exactly).
//
// A product that an error-free transformation adds must be rounded on its own.
// The assembler was seen to fuse a packed mul.rn with the packed add.rn that
// takes its result (sums of squares then came out with FP32 errors), which it
// does not do to the scalar instructions, so such products are written as
// fma(a, b, nz) with nz = {-0, -0} read from memory (a kernel argument): the
// same value, and nothing to fuse.  Plain mul2 is for products by powers of
// two and for low-order terms.
#pragma once
#include "cov_df.cuh"

namespace covgpu {

typedef unsigned long long f2;   // two FP32 values: low word, high word

__device__ __forceinline__ f2 pk2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 dup2(float a) { return pk2(a, a); }
__device__ __forceinline__ float2 un2(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// the rounded product; nz = {-0, -0} as the compiler cannot know it
__device__ __forceinline__ f2 mulr2(f2 a, f2 b, f2 nz) { return fma2(a, b, nz); }
__device__ __forceinline__ f2 neg2(f2 a) { return a ^ 0x8000000080000000ull; }

struct df2 { f2 hi, lo; };

__device__ __forceinline__ df2 dfz2() { return {0ull, 0ull}; }
__device__ __forceinline__ df2 dup_df(df a) { return {dup2(a.hi), dup2(a.lo)}; }
__device__ __forceinline__ df half_df(df2 a, int h) {
  const float2 x = un2(a.hi), y = un2(a.lo);
  return h ? df{x.y, y.y} : df{x.x, y.x};
}
__device__ __forceinline__ df2 two_sum2(f2 a, f2 b) {
  const f2 s = add2(a, b), bb = sub2(s, a);
  return {s, add2(sub2(a, sub2(s, bb)), sub2(b, bb))};
}
// a + b with b given negated (nb = -b)
__device__ __forceinline__ df2 two_sum2_n(f2 a, f2 nb) {
  const f2 s = sub2(a, nb), bb = sub2(s, a);
  return {s, sub2(sub2(a, sub2(s, bb)), add2(nb, bb))};
}
__device__ __forceinline__ df2 fast_two_sum2(f2 a, f2 b) {
  const f2 s = add2(a, b);
  return {s, sub2(b, sub2(s, a))};
}
__device__ __forceinline__ df2 df2_norm(df2 a) { return fast_two_sum2(a.hi, a.lo); }
__device__ __forceinline__ df2 df2_add_f(df2 a, f2 b) {
  const df2 s = two_sum2(a.hi, b);
  return fast_two_sum2(s.hi, add2(s.lo, a.lo));
}
__device__ __forceinline__ df2 df2_add(df2 a, df2 b) {
  const df2 s = two_sum2(a.hi, b.hi);
  return fast_two_sum2(s.hi, add2(s.lo, add2(a.lo, b.lo)));
}
// a + b where the short two_sum is exact (|a| >= |b|, or a = 0)
__device__ __forceinline__ df2 df2_add_fast(df2 a, df2 b) {
  const df2 s = fast_two_sum2(a.hi, b.hi);
  return fast_two_sum2(s.hi, add2(s.lo, add2(a.lo, b.lo)));
}
__device__ __forceinline__ df2 df2_sub(df2 a, df2 b) {
  const df2 s = two_sum2_n(a.hi, b.hi);
  return fast_two_sum2(s.hi, add2(s.lo, sub2(a.lo, b.lo)));
}
__device__ __forceinline__ void df2_acc(df2& s, df2 b) {
  const df2 t = two_sum2(s.hi, b.hi);
  s.hi = t.hi;
  s.lo = add2(s.lo, add2(t.lo, b.lo));
}
// a b left unnormalised, formed from -(a.hi b.hi); na = -a.hi
__device__ __forceinline__ df2 df2_mul_un(df2 a, f2 na, df2 b, f2 nz) {
  const f2 np = mulr2(na, b.hi, nz);
  return {neg2(np), fma2(a.hi, b.lo, fma2(a.lo, b.hi, fma2(a.hi, b.hi, np)))};
}
// s += a b, the product unnormalised; na = -a.hi
__device__ __forceinline__ void df2_acc_mul(df2& s, df2 a, f2 na, df2 b, f2 nz) {
  const f2 np = mulr2(na, b.hi, nz);                                  // -(a.hi b.hi), rounded
  const f2 lo = fma2(a.hi, b.lo, fma2(a.lo, b.hi, fma2(a.hi, b.hi, np)));
  const df2 t = two_sum2_n(s.hi, np);
  s.hi = t.hi;
  s.lo = add2(s.lo, add2(t.lo, lo));
}
__device__ __forceinline__ df2 df2_mul_u(df2 a, df2 b, f2 nz) {
  const f2 p = mulr2(a.hi, b.hi, nz);
  return {p, fma2(a.hi, b.lo, fma2(a.lo, b.hi, fma2(a.hi, b.hi, neg2(p))))};
}
__device__ __forceinline__ df2 df2_mul(df2 a, df2 b, f2 nz) { return df2_norm(df2_mul_u(a, b, nz)); }
// a^2, unnormalised; na = -a.hi
__device__ __forceinline__ df2 df2_sqr_u(df2 a, f2 na, f2 nz) {
  const f2 e = fma2(a.hi, a.hi, mulr2(na, a.hi, nz));
  return {mulr2(a.hi, a.hi, nz), fma2(add2(a.hi, a.hi), a.lo, e)};
}
__device__ __forceinline__ df2 df2_scale(df2 a, float s) { return {mul2(a.hi, dup2(s)), mul2(a.lo, dup2(s))}; }
// a/b and 1/b as df_div forms them
__device__ __forceinline__ df2 df2_div(df2 a, df2 b, f2 nz) {
  const float2 bh = un2(b.hi);
  const f2 r = pk2(1.0f / bh.x, 1.0f / bh.y);
  const f2 q = mulr2(a.hi, r, nz), np = mulr2(neg2(b.hi), q, nz);   // -(b.hi q), rounded
  // -(b q) normalised, then the residual a - b q
  const df2 pr = fast_two_sum2(np, neg2(fma2(b.lo, q, fma2(b.hi, q, np))));
  const df2 res = df2_add(a, pr);
  return fast_two_sum2(q, mulr2(res.hi, r, nz));
}
__device__ __forceinline__ df2 df2_recip(df2 b, f2 nz) { return df2_div({dup2(1.0f), 0ull}, b, nz); }

// df_log of both halves (cov_df.cuh), the table looked up per half.  What
// works on the table's values is scalar: a packed operation would first need
// its operands moved next to each other.
__device__ __forceinline__ df2 df2_log(df2 a, const float4* __restrict__ tab, f2 nz) {
  const float2 ah = un2(a.hi), al = un2(a.lo);
  float u[2], pe[2], rs[2], re[2], rl[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int bits = __float_as_int(h ? ah.y : ah.x);
    const float4 T = tab[(bits >> 16) & (LOGTAB_N - 1)];
    const float2 K = reinterpret_cast<const float2*>(tab + LOGTAB_N)[((unsigned)bits >> 23) & 255u];   // k ln 2
    const float m = __int_as_float((bits & 0x007FFFFF) | 0x3F800000);
    const float p = __fmul_rn(m, T.x);
    pe[h] = fmaf(m, T.x, -p);
    u[h] = __fsub_rn(p, 1.0f);   // exact (p within 2^-7 of 1)
    // k ln 2 - ln r_j: k ln 2 is 0 or the larger term, so two_sum in its short form
    rs[h] = __fadd_rn(K.x, T.y);
    re[h] = __fsub_rn(T.y, __fsub_rn(rs[h], K.x));
    rl[h] = __fadd_rn(K.y, T.z);
  }
  const df2 t = fast_two_sum2(pk2(u[0], u[1]), pk2(pe[0], pe[1]));
  const f2 nt = neg2(t.hi);
  const f2 ns2 = mulr2(nt, t.hi, nz);                              // -t^2, rounded
  const f2 s2e = fma2(t.hi, t.hi, ns2);
  const f2 poly = mulr2(mul2(nt, ns2), fma2(t.hi, fma2(t.hi, dup2(0.2f), dup2(-0.25f)), dup2(0.333333343f)), nz);
  const f2 corr = pk2(__fdividef(al.x, ah.x), __fdividef(al.y, ah.y));
  const f2 low = add2(fma2(dup2(-0.5f), s2e, fma2(nt, t.lo, t.lo)), add2(poly, corr));
  const df2 l1p = fast_two_sum2(t.hi, mul2(dup2(0.5f), ns2));
  const df2 r = fast_two_sum2(pk2(rs[0], rs[1]), add2(pk2(re[0], re[1]), pk2(rl[0], rl[1])));
  // ln(1 + t) is no larger than r, or of the other sign and near it (an exact sum)
  return df2_add_fast(r, {l1p.hi, add2(l1p.lo, low)});
}

}  // namespace covgpu
