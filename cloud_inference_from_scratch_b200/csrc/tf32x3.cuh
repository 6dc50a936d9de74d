// Products of float32 values on the tensor cores (mma.sync m16n8k8, kind tf32) as accurate as float32 sums.
//
// A value is hi + lo: hi rounded to the 11 bits of tf32, lo the exact rest, of which the tensor core takes the first 11 bits.
// A product is hi hi + (hi lo + lo hi); what is left out (lo lo, and the last bit of lo) is about 2^-24 of it, with either
// sign.  The tensor core cuts what it adds: the small terms have an accumulator of their own, or come first, and callers keep
// accumulators short (a few steps of 8) and add them up in registers.
//
// Values whose hi overflows, infinities and NaN are the caller's to find (`tf32_unsafe`) and to work out otherwise.
#pragma once

#include <stdint.h>

namespace cie {

struct Tf32Split { uint32_t hi, lo; };

__device__ __forceinline__ Tf32Split tf32_split(float x) {
  Tf32Split s;
  s.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  s.lo = __float_as_uint(x - __uint_as_float(s.hi));
  return s;
}
// Rounds to infinity, or is an infinity or NaN already.
__device__ __forceinline__ bool tf32_unsafe(float x) { return (__float_as_uint(x) & 0x7fffffffu) >= 0x7f7ff000u; }

// A 16 x 8 operand: rows g and g + 8, columns t and t + 4 of lane 4 g + t, in the instruction's order.
struct Tf32A {
  uint32_t hi[4], lo[4];
  __device__ __forceinline__ void set(int i, float x) {
    const Tf32Split s = tf32_split(x);
    hi[i] = s.hi;
    lo[i] = s.lo;
  }
};
// An 8 x 8 operand: rows t and t + 4 of column g.
struct Tf32B {
  uint32_t hi[2], lo[2];
  Tf32B() = default;
  __device__ __forceinline__ Tf32B(float x, float y) {
    const Tf32Split a = tf32_split(x), b = tf32_split(y);
    hi[0] = a.hi; hi[1] = b.hi;
    lo[0] = a.lo; lo[1] = b.lo;
  }
};

__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_tf32_first(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}

// A 16 x 8 sum: rows g and g + 8 (elements 0 1, 2 3), columns 2 t and 2 t + 1 of lane 4 g + t.
// kRounded: the large products of every step of 8 have an accumulator of their own and are added up in registers, where a sum is
// rounded and not cut.  Gated linear attention of portions of 333 tokens is 1.83e-7 of its norm from 64 bits so, 2.09e-7
// with one accumulator and 1.95e-7 on the CUDA cores (the gated delta rule 1.73, 1.83 and 1.91e-7; the generalized rule's
// 4.0e-7 against 4.8e-7 do without); 2,048 tokens, 16 heads of 128: 138 us, 134 with one.
template <bool kRounded>
struct Tf32Sum {
  float big[4], small[4];
  // `first`: a constant, true for the first product of the sum
  __device__ __forceinline__ void add(const Tf32A& a, const Tf32B& b, bool first) {
    if (first) {
      mma_tf32_first(small, a.lo, b.hi);
      mma_tf32_first(big, a.hi, b.hi);
    } else {
      mma_tf32(small, a.lo, b.hi);
      if (kRounded) {
        float more[4];
        mma_tf32_first(more, a.hi, b.hi);
#pragma unroll
        for (int i = 0; i < 4; ++i) big[i] += more[i];
      } else {
        mma_tf32(big, a.hi, b.hi);
      }
    }
    mma_tf32(small, a.hi, b.lo);
  }
  __device__ __forceinline__ float of(int i) const { return big[i] + small[i]; }
};

}  // namespace cie
