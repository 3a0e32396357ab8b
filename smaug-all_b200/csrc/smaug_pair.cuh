// smaug_pair.cuh -- two FP32 lanes in one 64-bit register pair, for the packed
// FP32 instructions of sm_100a (add/sub/mul/fma .rn.ftz.f32x2).
//
// Each lane is rounded exactly as the scalar instruction of the same name
// rounds it (round to nearest even, subnormals flushed as the -ftz=true build
// flushes them).  A product that goes into a sum is to be written with pfma:
// ptxas contracts a packed mul and the add behind it into one fma where it sees
// fit (measured: C - A * B and C + A * B differ from their scalar forms in one
// value of five), which it does not do to the scalar .rn forms.  Written so, a
// computation gives the same bits on one lane (f1) and on two.  Negation is a multiply by -1 (exact, and it
// keeps the sign of zero), since the packed fma has no negated operand form.
#pragma once

namespace SMAUG_NS {

struct f2 {
  unsigned long long r;
};

__device__ __forceinline__ f2 f2_make(float lo, float hi) {
  f2 o;
  asm("mov.b64 %0, {%1, %2};" : "=l"(o.r) : "f"(lo), "f"(hi));
  return o;
}
__device__ __forceinline__ f2 f2_splat(float a) { return f2_make(a, a); }
__device__ __forceinline__ float f2_lo(f2 x) {
  float lo;
  asm("{\n\t.reg .f32 h;\n\tmov.b64 {%0, h}, %1;\n\t}" : "=f"(lo) : "l"(x.r));
  return lo;
}
__device__ __forceinline__ float f2_hi(f2 x) {
  float hi;
  asm("{\n\t.reg .f32 l;\n\tmov.b64 {l, %0}, %1;\n\t}" : "=f"(hi) : "l"(x.r));
  return hi;
}
__device__ __forceinline__ f2 operator+(f2 a, f2 b) {
  f2 o;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(o.r) : "l"(a.r), "l"(b.r));
  return o;
}
__device__ __forceinline__ f2 operator-(f2 a, f2 b) {
  f2 o;
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(o.r) : "l"(a.r), "l"(b.r));
  return o;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b) {
  f2 o;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(o.r) : "l"(a.r), "l"(b.r));
  return o;
}
// a * b + c with one rounding per lane
__device__ __forceinline__ f2 pfma(f2 a, f2 b, f2 c) {
  f2 o;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(o.r) : "l"(a.r), "l"(b.r), "l"(c.r));
  return o;
}
__device__ __forceinline__ f2 pneg(f2 a) { return a * f2_splat(-1.0f); }

// One lane with the same operations, as instructions the compiler leaves alone
// too, so that each is rounded as a lane of f2 rounds it.
struct f1 {
  float r;
};
__device__ __forceinline__ f1 operator+(f1 a, f1 b) {
  f1 o;
  asm("add.rn.ftz.f32 %0, %1, %2;" : "=f"(o.r) : "f"(a.r), "f"(b.r));
  return o;
}
__device__ __forceinline__ f1 operator-(f1 a, f1 b) {
  f1 o;
  asm("sub.rn.ftz.f32 %0, %1, %2;" : "=f"(o.r) : "f"(a.r), "f"(b.r));
  return o;
}
__device__ __forceinline__ f1 operator*(f1 a, f1 b) {
  f1 o;
  asm("mul.rn.ftz.f32 %0, %1, %2;" : "=f"(o.r) : "f"(a.r), "f"(b.r));
  return o;
}
__device__ __forceinline__ f1 pfma(f1 a, f1 b, f1 c) {
  f1 o;
  asm("fma.rn.ftz.f32 %0, %1, %2, %3;" : "=f"(o.r) : "f"(a.r), "f"(b.r), "f"(c.r));
  return o;
}
__device__ __forceinline__ f1 pneg(f1 a) { return {-a.r}; }

// Common names of both: all lanes alike, a value per lane (f1 takes the
// first), a lane, and zero in the lanes whose flag is off.
template <typename P>
__device__ __forceinline__ P splat(float a);
template <>
__device__ __forceinline__ f1 splat<f1>(float a) {
  return {a};
}
template <>
__device__ __forceinline__ f2 splat<f2>(float a) {
  return f2_splat(a);
}
template <typename P>
__device__ __forceinline__ P pack(float lo, float hi);
template <>
__device__ __forceinline__ f1 pack<f1>(float lo, float) {
  return {lo};
}
template <>
__device__ __forceinline__ f2 pack<f2>(float lo, float hi) {
  return f2_make(lo, hi);
}
__device__ __forceinline__ float lane(f1 x, int) { return x.r; }
__device__ __forceinline__ float lane(f2 x, int k) { return k ? f2_hi(x) : f2_lo(x); }
template <typename P>
__device__ __forceinline__ P keep(bool lo, bool hi, P x) {
  return pack<P>(lo ? lane(x, 0) : 0.0f, hi ? lane(x, 1) : 0.0f);
}

}  // namespace SMAUG_NS
