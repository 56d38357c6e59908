// pair.cuh -- two float32 values in one instruction.
//
// sm_100a's packed single-precision add, subtract, multiply and fused multiply-add round
// each half as the scalar instruction does and take one issue slot for two results.
// Included inside the arithmetic namespace; both builds get exactly the operations written
// (nothing is contracted).
#pragma once

struct F2 {
  float x, y;
};
#define RB_PAIR_OP(name, op)                                                                             \
  __device__ __forceinline__ F2 name(F2 a, F2 b) {                                                       \
    F2 r;                                                                                                \
    asm("{.reg .b64 a, b, r; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; " op " r, a, b; mov.b64 {%0, %1}, r;}" \
        : "=f"(r.x), "=f"(r.y)                                                                           \
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                       \
    return r;                                                                                            \
  }
RB_PAIR_OP(operator+, "add.rn.f32x2")
RB_PAIR_OP(operator-, "sub.rn.f32x2")
RB_PAIR_OP(operator*, "mul.rn.f32x2")
#undef RB_PAIR_OP
__device__ __forceinline__ F2 both(float v) { return F2{v, v}; }
__device__ __forceinline__ F2 operator*(float a, F2 b) { return both(a) * b; }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("{.reg .b64 a, b, c, r; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 c, {%6, %7}; "
      "fma.rn.f32x2 r, a, b, c; mov.b64 {%0, %1}, r;}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}

// a + b and a - b where an operand is a product: as multiply-adds by a one that the
// assembler cannot see, since it contracts a packed product into the packed sum that uses
// it, whatever rounding the two instructions name.
__constant__ float c_pair_one = 1.0f;
struct PairOne {
  F2 plus, minus;
  __device__ __forceinline__ PairOne() {
    const float one = c_pair_one;
    plus = both(one);
    minus = both(-one);
  }
  __device__ __forceinline__ F2 add(F2 a, F2 b) const { return fma2(a, plus, b); }
  __device__ __forceinline__ F2 sub(F2 a, F2 b) const { return fma2(b, minus, a); }
};
