// Two float32 lanes in one register pair (add, subtract, multiply and FMA of
// sm_100 and later: one instruction for both lanes, each rounded as the scalar
// instruction rounds it).  Measured on this card: 64 lane pairs per clock and SM,
// the same lanes as the scalar forms for half the issue slots.
//
// An f2_add of two f2_mul results is contracted to an FMA by the assembler in
// spite of its .rn (seen on 25 % of random operands with CUDA 13.0; an f2_add of
// one product and something else is not): add such products lane by lane.
#pragma once

#include "common.cuh"

namespace gg {

struct F2 {
  unsigned long long v = 0;  // both lanes +0
};

__device__ __forceinline__ F2 f2(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ void f2_split(F2 a, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// a - b as b * -1 + a, rounded once like the subtraction: the packed add has no
// negated operands, and flipping the signs costs two more instructions.
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { return f2_fma(b, f2(-1.0f), a); }

__device__ __forceinline__ float f2_sum(F2 a) {
  float x, y;
  f2_split(a, x, y);
  return __fadd_rn(x, y);
}

// Knuth TwoSum of both lanes: s + e == a + b exactly.
__device__ __forceinline__ void f2_two_sum(F2 a, F2 b, F2& s, F2& e) {
  s = f2_add(a, b);
  const F2 bb = f2_sub(s, a);
  e = f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb));
}

// Two float-float accumulators.
struct FF2 {
  F2 hi, lo;
  __device__ __forceinline__ void add(F2 x) {
    F2 s, e;
    f2_two_sum(hi, x, s, e);
    hi = s;
    lo = f2_add(lo, e);
  }
  // Both lanes in one float-float sum.
  __device__ __forceinline__ FF merged() const {
    float ah, bh, al, bl;
    f2_split(hi, ah, bh);
    f2_split(lo, al, bl);
    FF r;
    float e;
    two_sum(ah, bh, r.hi, e);
    r.lo = __fadd_rn(__fadd_rn(al, bl), e);
    return r;
  }
};

// Float-float sums of two sequences and of their squares: FF::add and
// FF::add_prod in packed instructions, each rounded alike.  Zeros change
// nothing.
struct F2Moments {
  FF2 first;
  F2 hi, lo;  // of the squares
  __device__ __forceinline__ void add(F2 x) {
    first.add(x);
    const F2 np = f2_mul(x, f2_mul(x, f2(-1.0f)));  // -(x * x)
    const F2 pe = f2_fma(x, x, np);                 // its rounding error
    const F2 s = f2_sub(hi, np);
    const F2 b = f2_sub(s, hi);
    const F2 e = f2_sub(f2_sub(hi, f2_sub(s, b)), f2_add(np, b));
    hi = s;
    lo = f2_add(f2_add(lo, e), pe);
  }
  // (sum, sum of squares) of the two sequences
  __device__ __forceinline__ void split(FF& s1, FF& s2, FF& t1, FF& t2) const {
    f2_split(first.hi, s1.hi, t1.hi);
    f2_split(first.lo, s1.lo, t1.lo);
    f2_split(hi, s2.hi, t2.hi);
    f2_split(lo, s2.lo, t2.lo);
  }
};

}  // namespace gg
