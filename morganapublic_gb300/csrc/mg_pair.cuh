// Two elements per thread: packed pairs of floats (f2) and of double-words (ff2).
//
// sm_103a issues one packed instruction (add / sub / mul / fma .rn.f32x2) for two
// FP32 lane operations at the full 128 lanes per SM per clock (measured: 122-127
// lane operations per clock for packed and scalar alike).  The element kernels
// are bound by instruction issue, so the pair form halves their arithmetic
// instructions.  Each lane is the IEEE operation of its scalar form; the
// double-word algorithms are those of mg_ff.cuh, with the low-order terms
// chained through FMAs.
#pragma once

#include "mg_ff.cuh"

namespace mg {

struct f2 {
  unsigned long long v;  // lanes x (low word) and y
};

__device__ __forceinline__ f2 f2_make(float x, float y)
{
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 f2_get(f2 a)
{
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
  return r;
}
__device__ __forceinline__ f2 operator+(f2 a, f2 b)
{
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 operator-(f2 a, f2 b)
{
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b)
{
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ f2 operator-(f2 a) { return f2{a.v ^ 0x8000000080000000ull}; }

// Reciprocal estimate of both lanes (MUFU.RCP, relative error ~2^-23, subnormals
// flushed) with one Newton step.
__device__ __forceinline__ f2 f2_rcp(f2 b)
{
  const float2 d = f2_get(b);
  float x, y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(d.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d.y));
  const f2 r = f2_make(x, y);
  return fma2(r, fma2(-b, r, f2_make(1.0f, 1.0f)), r);
}

// a b - c d with the rounding error of c d added back (Kahan), nc = -c: within 1.5
// ulp however much the products cancel
__device__ __forceinline__ f2 f2_cross(f2 a, f2 b, f2 c, f2 d, f2 nc)
{
  const f2 nw = nc * d;
  return fma2(a, b, nw) - fma2(c, d, nw);
}

struct ff2 {
  f2 hi, lo;
};

__device__ __forceinline__ ff2 ff2_make(ff x, ff y) { return ff2{f2_make(x.hi, y.hi), f2_make(x.lo, y.lo)}; }
__device__ __forceinline__ ff2 operator-(ff2 a) { return ff2{-a.hi, -a.lo}; }

// hi + lo with |hi| >= |lo| (or hi = 0), renormalised
__device__ __forceinline__ ff2 f2_fast_two_sum(f2 a, f2 b)
{
  const f2 s = a + b;
  return ff2{s, b - (s - a)};
}
// error-free sum and difference
__device__ __forceinline__ ff2 f2_two_sum(f2 a, f2 b)
{
  const f2 s = a + b, bb = s - a;
  return ff2{s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ ff2 f2_two_diff(f2 a, f2 b)
{
  const f2 s = a - b, bb = a - s;  // bb: the part of b in s
  return ff2{s, (a - (s + bb)) + (bb - b)};
}

// a b - c d of double-words, renormalised; na, nc, nd hold -a.hi, -c.hi, -d.hi.
// The product errors come out negated (fma(-a, b, a b rounded)), which costs no
// sign flip: ab = p - pe, cd = q - qe.
__device__ __forceinline__ ff2 ff2_cross(ff2 a, ff2 b, ff2 c, ff2 d, f2 na, f2 nc, f2 nd)
{
  const f2 p = a.hi * b.hi, pe = fma2(na, b.hi, p);
  const f2 q = c.hi * d.hi, qe = fma2(nc, d.hi, q);
  const ff2 s = f2_two_diff(p, q);
  const f2 x = fma2(a.lo, b.hi, fma2(a.hi, b.lo, s.lo));
  const f2 y = fma2(c.lo, nd, fma2(nc, d.lo, qe - pe));
  return f2_fast_two_sum(s.hi, x + y);
}

// a . b of double-word 3-vectors, na[k] = -a[k].hi; not renormalised: |lo| is a few
// 2^-24 of the largest term
__device__ __forceinline__ ff2 ff2_dot3(const ff2* a, const ff2* b, const f2* na)
{
  f2 hi = a[0].hi * b[0].hi;
  f2 lo = fma2(a[0].lo, b[0].hi, a[0].hi * b[0].lo) - fma2(na[0], b[0].hi, hi);
#pragma unroll
  for (int k = 1; k < 3; ++k) {
    const f2 q = a[k].hi * b[k].hi, qe = fma2(na[k], b[k].hi, q);
    const ff2 s = f2_two_sum(hi, q);
    hi = s.hi;
    lo = lo + fma2(a[k].hi, b[k].lo, fma2(a[k].lo, b[k].hi, s.lo - qe));
  }
  return ff2{hi, lo};
}

}  // namespace mg
