// rb_common.cuh -- shared device helpers for the river-basin solver kernels.
//
// Two arithmetic contracts, one source:
//  * exact (every translation unit in csrc/): compiled with --fmad=false and IEEE
//    division / square root, so each operation rounds once in the reference's
//    expression order (identical to the CPU oracle); the fractional powers come
//    from include/rb_detmath.h;
//  * fast (csrc/fast/, RB_FAST_MATH defined, everything in namespace rb::fast):
//    contracted multiply-adds and the hardware's approximate division, square root
//    and powers -- the arithmetic of a GPU build of the reference, held to the solver
//    tolerance instead of bit equality. Compensated (Kahan) additions stay explicit
//    IEEE adds in both.
// `rmax/rmin/rclamp` are the scalar builtins of the reference's kernel language
// (a > b ? a : b, a < b ? a : b, min(max(lo,x),hi)), which differ from
// fmaxf/fminf on signed zeros.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "rb_detmath.h"
#include "rbsim.h"

// The kernels of a translation unit live in rb (exact) or rb::fast (fast).
#if defined(RB_FAST_MATH)
#define RB_ARITH_BEGIN namespace fast {
#define RB_ARITH_END }
#else
#define RB_ARITH_BEGIN
#define RB_ARITH_END
#endif

namespace rb {

constexpr float kG = 9.81f;     // solver/core/grid.py:43 GRAVITY
constexpr float kHDry = 1.0e-3f;  // solver/core/grid.py:48 H_DRY

RB_ARITH_BEGIN

__device__ __forceinline__ float rmax(float a, float b) { return a > b ? a : b; }
__device__ __forceinline__ float rmin(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float rclamp(float x, float lo, float hi) { return rmin(rmax(lo, x), hi); }

// sources.py:66-82 kahan_add: (total, comp) <- compensated total + inc. Explicit
// IEEE adds, which no build contracts or reassociates.
__device__ __forceinline__ void kahan_add(float& total, float& comp, float inc) {
  const float y = __fsub_rn(inc, comp);
  const float t = __fadd_rn(total, y);
  comp = __fsub_rn(__fsub_rn(t, total), y);
  total = t;
}

#if defined(RB_FAST_MATH)
// Fast arithmetic: the approximate division has no slow path to steer around, so
// the quotient helpers are plain divisions (an unused lane divides by 1).
__device__ __forceinline__ float opaque(float v) { return v; }
__device__ __forceinline__ float div_pos(float x, float y) { return x / y; }
__device__ __forceinline__ float div_if(bool use, float x, float y) { return use ? x / (use ? y : 1.0f) : 0.0f; }
__device__ __forceinline__ float div_in_branch(float x, float y) { return x / y; }
// x / g
__device__ __forceinline__ float div_g(float x) { return x * (1.0f / kG); }
// A quotient as x times the reciprocal unit's approximation: within 2^-22 of x / y for
// |y| in [2^-60, 2^60] (the unit is documented to an ulp, the product rounds once more).
__device__ __forceinline__ float rcp_near(float y) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return r;
}
// The square-root unit: within 2^-23 for a normal x (as documented), 0 for a subnormal.
__device__ __forceinline__ float sqrt_near(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// h^(7/3) for h in [H_DRY, 2^20] as 2^(p log2 h) on the logarithm and exponential units.
// With their documented errors (2^-22 of max(1, |log2 h|), and 2 ulp) the relative error
// is below ln 2 (p 2^-22 max(1, |log2 h|) + 2^-24 |p log2 h|) + 2^-22 + 2^-24. The power
// is above 2^-24 there, so that the maximum changes no value; without it the power and the
// reciprocal that callers take of it came out an ulp apart from the two taken one by one.
__device__ __forceinline__ float pow73_near(float h) {
  float l, e;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(h));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(2.33333325f * l));
  return fmaxf(e, 0x1p-24f);
}
// n / d >= 0 for |d| > 0, from the signs
__device__ __forceinline__ bool quotient_nonneg(float n, float d) { return n == 0.0f || ((n > 0.0f) == (d > 0.0f)); }
// x ^ float32(p) for x > 0 with the float32 exponents of the reference (7/3, 1/3, 4/3, 1.5)
__device__ __forceinline__ float pow73(float x) { return __powf(x, 2.33333325f); }
__device__ __forceinline__ float pow13(float x) { return __powf(x, 0.333333343f); }
__device__ __forceinline__ float pow43(float x) { return __powf(x, 1.33333337f); }
__device__ __forceinline__ float pow15(float x) { return x * sqrtf(x); }
#else
// Zero operands. The IEEE single-precision division takes its slow path when the
// dividend is zero (about 3x the cost of the fast path on B200) or the divisor is.
// Still water, dry neighbours and frictionless beds make such operands common, and
// a guard in the source does not keep them away: the compiler evaluates a guarded
// division unconditionally and selects the result, so a discarded quotient of a
// dry cell still pays the slow path. The helpers below give the division 1 in place of an
// operand that would send it down the slow path, and select the exact result
// themselves (0 / y = 0 with the dividend's sign for y > 0).
// `opaque` hides the substituted operand from the optimizer, which would otherwise
// fold the two selects back into the original division; the move itself compiles to
// nothing.
__device__ __forceinline__ float opaque(float v) {
  float r;
  asm("mov.b32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// x / y, bit for bit, for any x and y.
__device__ __forceinline__ float div_pos(float x, float y) {
  const bool same = x == 0.0f && y > 0.0f;  // the quotient is x itself
  const float q = opaque(same ? 1.0f : x) / y;
  return same ? x : q;
}

// use ? x / y : 0, where the division of an unused lane divides by 1 (its divisor,
// e.g. the depth of a dry cell, may be 0).
__device__ __forceinline__ float div_if(bool use, float x, float y) {
  const float q = div_pos(x, opaque(use ? y : 1.0f));
  return use ? q : 0.0f;
}

// The IEEE quotient x / y as inline PTX, which the compiler cannot evaluate ahead
// of the branch that guards it: for divisions that a data-dependent branch is meant
// to skip, where an ordinary '/' would be computed for every lane regardless.
__device__ __forceinline__ float div_in_branch(float x, float y) {
  float q;
  asm volatile("div.rn.f32 %0, %1, %2;" : "=f"(q) : "f"(x), "f"(y));
  return q;
}

// The IEEE quotient a / b without a slow path, for operands inside a safe range: a
// reciprocal approximation sharpened by one Newton step and a residual correction, all
// in fused multiply-adds (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990: with y the correctly
// rounded 1 / b and q0 within an ulp of a / b, RN(q0 + y RN(a - b q0)) is the correctly
// rounded quotient). One Newton step on this GPU's approximation gives that y for every
// b in [2^-24, 2^64] (tests/test_gpu_arith_sweep.py compares all of them, and the other
// ranges named here, with the IEEE operations). Over the same b the quotient is exact in
// this sense for |a| in [2^-60, 2^60] or a = 0 (div_rn_small_ok checks the lower end): it
// stays above 2^-124, and its residual, a multiple of 2^-107 or more, does not underflow.
// Outside, the result is unspecified, but for b >= 2^-24 never above 2^-35 where |a| <
// 2^-60; a NaN a gives NaN.
__device__ __forceinline__ bool div_rn_small_ok(float a) { return (a == 0.0f) | !(fabsf(a) < 0x1p-60f); }
// a / b given y, the correctly rounded 1 / b, for b > 0: the sign is the dividend's, also
// that of a zero.
__device__ __forceinline__ float div_rn_by(float a, float b, float y) {
  const float q0 = a * y;
  const float q = __fmaf_rn(__fmaf_rn(-b, q0, a), y, q0);
  return __uint_as_float((__float_as_uint(q) & 0x7fffffffu) | (__float_as_uint(a) & 0x80000000u));
}
__device__ __forceinline__ float rcp_rn(float b) {  // the correctly rounded 1 / b, b in [2^-24, 2^64]
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
  return __fmaf_rn(__fmaf_rn(-b, y, 1.0f), y, y);
}
__device__ __forceinline__ float div_rn(float a, float b) { return div_rn_by(a, b, rcp_rn(b)); }

// The IEEE square root for a in [2^-100, 2^100]: Markstein's residual correction of
// a * rsqrt(a) (same paper).
__device__ __forceinline__ float sqrt_rn(float a) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a));
  const float q = a * y;
  return __fmaf_rn(__fmaf_rn(-q, q, a), 0.5f * y, q);
}

// rb_pow73f for x in [2^-12, 2^20], the same bits without a branch. The operations of
// include/rb_detmath.h on x scaled by 2^(-3q) into [1, 8), q = floor(e / 3): scaling by
// a power of two commutes with every rounding here (all values stay normal), so the
// factors 2^q and 2^(3q) of the cube root and of x^2 become one exponent of the result.
__device__ __forceinline__ float pow73_mid(float x) {
  const unsigned b = __float_as_uint(x);
  const int k = (int)(b >> 23) - 115;  // e + 12 in [0, 32]
  const int q = (k * 43) >> 7;         // floor(k / 3); e = k - 12, so floor(e / 3) = q - 4
  const int r = k - 3 * q;
  const unsigned mb = (b & 0x007fffffu) | 0x3f800000u;
  const float m = __uint_as_float(mb), tf = __uint_as_float(mb + ((unsigned)r << 23));
  float w = ((-0.0488736666738987f * m + 0.3129411041736603f) * m - 0.8028873205184937f) * m + 1.5385289192199707f;
  w = w * (r == 0 ? 1.0f : (r == 1 ? 0.7937005162239075f : 0.6299605369567871f));
  w = w + w * ((1.0f - tf * ((w * w) * w)) * 0.333333343f);
  const double t = (double)tf;
  double wd = (double)w;
  wd = wd + wd * ((1.0 - t * ((wd * wd) * wd)) * 0.3333333333333333);
  const float t1 = m - 1.0f;
  const float log2m = ((((0.04392862692475319f * t1 - 0.18983244895935059f) * t1 + 0.4115614891052246f) * t1 -
                        0.7072534561157227f) * t1 + 1.4415920972824097f) * t1 + 1.4390930118679535e-05f;
  const float ef = __uint_as_float(0x4b000000u + (unsigned)k) - 8388620.0f;  // (float)(k - 12)
  const double u = RB_DELTA_73 * (double)((ef + log2m) * 0.693147182f);
  const double v = ((t * t) * (t * (wd * wd))) * ((1.0 - u) + 0.5 * (u * u));
  return __uint_as_float(__float_as_uint((float)v) + ((unsigned)(7 * (q - 4)) << 23));
}

__device__ __forceinline__ float div_g(float x) { return rb_div_g(x); }  // x / g, bit for bit
// rb_div_g for x >= 2^-99, without its other branch
__device__ __forceinline__ float rb_div_g_mid(float x) {
  return __fmaf_rn(x, 0x1.a1887ap-4f, x * 0x1.dcb5p-38f);
}
__device__ __forceinline__ bool quotient_nonneg(float n, float d) { return rb_quotient_nonneg(n, d) != 0; }
__device__ __forceinline__ float pow73(float x) { return rb_pow73f(x); }
__device__ __forceinline__ float pow13(float x) { return rb_pow13f(x); }
__device__ __forceinline__ float pow43(float x) { return rb_pow43f(x); }
__device__ __forceinline__ float pow15(float x) { return rb_pow15f(x); }
#endif  // RB_FAST_MATH

// channels.py:58-70 eta_subgrid: the storage curve h -> eta.
__device__ __forceinline__ float eta_subgrid(float h, float z, float w, float d, float dx) {
  float eta = h + z;
  if (w > 0.0f && d > 0.0f) {
    const float h_bf = div_pos(w * d, dx);
    if (h <= h_bf)
      eta = z - d + div_pos(h * dx, opaque(w > 0.0f ? w : 1.0f));
    else
      eta = z + (h - h_bf);
  }
  return eta;
}

// channels.py:73-83 column_depth: the water column that sets the wave speed.
__device__ __forceinline__ float column_depth(float h, float w, float d, float dx) {
  float col = h;
  if (w > 0.0f && d > 0.0f) {
    const float h_bf = div_pos(w * d, dx);
    if (h <= h_bf)
      col = div_pos(h * dx, opaque(w > 0.0f ? w : 1.0f));
    else
      col = d + (h - h_bf);
  }
  return col;
}

// friction.py:18-31 manning_denominator
__device__ __forceinline__ float manning_denominator(float q_prev, float h_flow, float n, float g, float dt) {
  return 1.0f + g * dt * n * n * fabsf(q_prev) / pow73(h_flow);
}

// num / manning_denominator(q_prev, h_flow, n, g, dt) for h_flow >= H_DRY, with the same
// bits. Where the friction numerator f = g dt n^2 |q_prev| is +0 or below 2^-60 the
// denominator is exactly 1 (h^(7/3) > 2^-24) and the quotient the numerator.
#if defined(RB_FAST_MATH)
__device__ __forceinline__ float manning_divide(float num, float q_prev, float h_flow, float n, float g, float dt) {
  const float f = g * dt * n * n * fabsf(q_prev);
  return num * rcp_near(1.0f + f * rcp_near(pow73_near(h_flow)));
}
#else
__device__ __forceinline__ float manning_divide_any(float num, float f, float h_flow) {
  if (f == 0.0f) return num;
  return div_pos(num, 1.0f + f / pow73(h_flow));
}
// The quick divisions and power inside their ranges, the general ones outside.
__device__ __forceinline__ float manning_divide(float num, float q_prev, float h_flow, float n, float g, float dt) {
  const float f = g * dt * n * n * fabsf(q_prev);
  float q = num;
  if (!(f < 0x1p-60f)) {
    const float den = 1.0f + div_rn(f, pow73_mid(h_flow));
    q = div_rn(num, den);
    const bool ok = (h_flow <= 0x1p19f) & (f <= 0x1p40f) & (den <= 0x1p20f) & div_rn_small_ok(num) &
                    !(fabsf(num) > 0x1p60f);
    if (!ok) q = manning_divide_any(num, f, h_flow);
  }
  return q;
}
#endif

// The reciprocal of dx a kernel's surface slopes multiply by, 0 where it must divide.
__device__ __forceinline__ float slope_rcp(float dx) {
#if defined(RB_FAST_MATH)
  return rcp_near(dx);
#else
  return dx >= 0x1p-20f && dx <= 0x1p20f ? 1.0f / dx : 0.0f;
#endif
}
// de / dx with rdx = slope_rcp(dx), the same bits.
__device__ __forceinline__ float face_slope(float de, float dx, float rdx) {
#if defined(RB_FAST_MATH)
  return de * rdx;
#else
  const float q = div_rn_by(de, dx, rdx);
  if (rdx == 0.0f || !div_rn_small_ok(de) || fabsf(de) > 0x1p60f) return div_in_branch(de, dx);
  return q;
#endif
}

// Float key whose unsigned order is the float order for values >= 0.
// Reductions here start from 0 (the reference zeroes its h_max slot before the
// atomic max), so only non-negative values are ever compared.
__device__ __forceinline__ unsigned int max_key(float v) { return __float_as_uint(v > 0.0f ? v : 0.0f); }

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Fixed-order warp sum (a butterfly tree; every lane ends with the same value).
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide max of non-negative values folded into *key with one atomic per block.
template <int NT>
__device__ __forceinline__ void block_max_to(float v, unsigned int* key, float* s_warp) {
  v = warp_max(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) s_warp[w] = v;
  __syncthreads();
  if (w == 0) {
    float x = l < NT / 32 ? s_warp[l] : 0.0f;
    x = warp_max(x);
    if (l == 0) atomicMax(key, max_key(x));
  }
}

// Block-wide f64 sum in a fixed order; the result is valid in thread 0.
template <int NT>
__device__ __forceinline__ double block_sum(double v, double* s_warp) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) s_warp[w] = v;
  __syncthreads();
  double x = 0.0;
  if (w == 0) {
    x = l < NT / 32 ? s_warp[l] : 0.0;
    x = warp_sum(x);
  }
  return x;
}

// Kahan-accumulate one tile's per-step f64 contribution into its ledger slot
// (slot[0] = running total, slot[1] = compensation). One writer per slot.
__device__ __forceinline__ void ledger_add(double* slot, double inc) {
  const double y = inc - slot[1];
  const double t = slot[0] + y;
  slot[1] = (t - slot[0]) - y;
  slot[0] = t;
}

__device__ __forceinline__ void flag_error(unsigned int* err, unsigned int bit) {
  if (err) atomicOr(err, bit);
}

RB_ARITH_END

// Programmatic dependent launch of the step chain (plan -> stage 1 -> stage 2 ->
// plan ..., or plan -> LI step -> plan ...). Each kernel of the chain waits until the
// kernel before it has completed with its memory visible, before it reads anything, and
// lets the next one be scheduled (pdl_trigger) once its work but for the reductions is
// done. Triggered at its start instead, the next grid's blocks take slots beside it and are
// packed onto few SMs (us per step, trigger at the start / at the end: 512^2 rain-on-grid
// 20.7 / 16.1, 256^2 dam break 30.8 / 23.1, 2048^2 dam break fast 192.1 / 190.3). The
// plan, one warp, triggers at its start. A kernel launched without the attribute does not
// start early, and for it the wait returns at once.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Whether the step chain is launched with programmatic stream serialization
// (default on; RBSIM_PDL=0 in the environment turns it off, for comparison).
bool pdl_enabled();

// Launch a kernel of the step chain, with the programmatic-serialization attribute
// when pdl_enabled(). The kernel must begin with pdl_wait().
template <class... Params, class... Args>
cudaError_t launch_chain(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                         Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Args&&>(args)...);
}
}  // namespace rb
