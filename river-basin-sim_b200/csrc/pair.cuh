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

#if !defined(RB_FAST_MATH)
// The steps of div_rn, rcp_rn, sqrt_rn and pow73_mid (rb_common.cuh) on both halves, the
// same bits over the same ranges. What is negated spares the negations of a residual
// (rounding is symmetric).
__device__ __forceinline__ F2 div_rn_by2(F2 a, F2 b, F2 ny) {  // ny = -1 / b, rounded once
  const F2 nq0 = a * ny;
  const F2 nq = fma2(fma2(b, nq0, a), ny, nq0);
  return F2{__uint_as_float((__float_as_uint(nq.x) & 0x7fffffffu) | (__float_as_uint(a.x) & 0x80000000u)),
            __uint_as_float((__float_as_uint(nq.y) & 0x7fffffffu) | (__float_as_uint(a.y) & 0x80000000u))};
}
__device__ __forceinline__ F2 neg_rcp_rn2(F2 b) {
  F2 y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(-b.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(-b.y));
  return fma2(fma2(b, y, both(1.0f)), y, y);
}
__device__ __forceinline__ F2 pow73_mid2(F2 x, const PairOne& one) {
  int kx, ky, qx, qy, rx, ry;
  F2 m, tf;
  auto split = [](float x, int& k, int& q, int& r, float& m, float& tf) {
    const unsigned b = __float_as_uint(x);
    k = (int)(b >> 23) - 115;
    q = (k * 43) >> 7;
    r = k - 3 * q;
    const unsigned mb = (b & 0x007fffffu) | 0x3f800000u;
    m = __uint_as_float(mb);
    tf = __uint_as_float(mb + ((unsigned)r << 23));
  };
  split(x.x, kx, qx, rx, m.x, tf.x);
  split(x.y, ky, qy, ry, m.y, tf.y);
  F2 w = one.add(both(-0.0488736666738987f) * m, both(0.3129411041736603f));
  w = one.add(w * m, both(-0.8028873205184937f));
  w = one.add(w * m, both(1.5385289192199707f));
  auto scale = [](int r) { return r == 0 ? 1.0f : (r == 1 ? 0.7937005162239075f : 0.6299605369567871f); };
  w = w * F2{scale(rx), scale(ry)};
  w = one.add(w, w * (one.sub(both(1.0f), tf * (w * w * w)) * both(0.333333343f)));
  const F2 t1 = m - both(1.0f);
  F2 l = one.add(both(0.04392862692475319f) * t1, both(-0.18983244895935059f));
  l = one.add(l * t1, both(0.4115614891052246f));
  l = one.add(l * t1, both(-0.7072534561157227f));
  l = one.add(l * t1, both(1.4415920972824097f));
  l = one.add(l * t1, both(1.4390930118679535e-05f));
  auto ef = [](int k) { return __uint_as_float(0x4b000000u + (unsigned)k) - 8388620.0f; };
  const F2 ln = (F2{ef(kx), ef(ky)} + l) * both(0.693147182f);
  auto finish = [](float tf, float wf, float ln, int q) {
    const double t = (double)tf;
    double wd = (double)wf;
    wd = wd + wd * ((1.0 - t * ((wd * wd) * wd)) * 0.3333333333333333);
    const double u = RB_DELTA_73 * (double)ln;
    const double v = ((t * t) * (t * (wd * wd))) * ((1.0 - u) + 0.5 * (u * u));
    return __uint_as_float(__float_as_uint((float)v) + ((unsigned)(7 * (q - 4)) << 23));
  };
  return F2{finish(tf.x, w.x, ln.x, qx), finish(tf.y, w.y, ln.y, qy)};
}
// -sqrt_rn of both halves, given them negated.
__device__ __forceinline__ F2 neg_sqrt_rn2(F2 na) {
  F2 y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.x) : "f"(-na.x));
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y.y) : "f"(-na.y));
  const F2 nq = na * y;
  return fma2(fma2(nq, nq, na), 0.5f * y, nq);
}
#endif
