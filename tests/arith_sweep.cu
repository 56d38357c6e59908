// arith_sweep.cu -- the step kernels' hand-written arithmetic (csrc/rb_common.cuh,
// csrc/pair.cuh, csrc/hllc_face.cuh) over the ranges its comments state. Compiled by test_gpu_arith_sweep.py
// once per arithmetic, with that build's flags. A check maps an index to operands and says
// whether what it got is what it should be.
#include <cfloat>
#include <cmath>

#include "rb_common.cuh"

namespace rb {
RB_ARITH_BEGIN
#include "pair.cuh"
#include "warp_stream.cuh"
#include "hllc_face.cuh"

using u64 = unsigned long long;

struct Operands {
  float a, b;
};
__device__ __forceinline__ unsigned bits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ float flt(unsigned u) { return __uint_as_float(u); }
__device__ __forceinline__ bool same(float x, float y) { return bits(x) == bits(y) || (x != x && y != y); }
__device__ __forceinline__ u64 mix(u64 x) {  // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
// 2^e, -126 <= e <= 127, and a float of that binade with the mantissa of `r`
__host__ __device__ constexpr unsigned pow2_bits(int e) { return (unsigned)(e + 127) << 23; }
__device__ __forceinline__ float in_binade(int e, unsigned r) { return flt(pow2_bits(e) | (r & 0x007fffffu)); }

// Operand pairs: `per` samples for each exponent ea in [ea0, ea1) of a and eb in [eb0, eb1)
// of b.
struct Pairs {
  int ea0, ea1, eb0, eb1;
  u64 per;
  __host__ __device__ u64 count() const { return (u64)(ea1 - ea0) * (u64)(eb1 - eb0) * per; }
  __device__ void at(u64 k, int& ea, int& eb, u64& r) const {
    const u64 pair = k / per;
    ea = ea0 + (int)(pair % (u64)(ea1 - ea0));
    eb = eb0 + (int)(pair / (u64)(ea1 - ea0));
    r = mix(k);
  }
};

#if !defined(RB_FAST_MATH)
// Every float of [2^lo, 2^hi]; the packed form's other half takes them in reverse.
template <int LO, int HI>
struct Every {
  static constexpr unsigned first = pow2_bits(LO), last = pow2_bits(HI);
  static u64 count() { return (u64)(last - first) + 1; }
  __device__ static float at(u64 k) { return flt(first + (unsigned)k); }
  __device__ static float mirror(u64 k) { return flt(last - (unsigned)k); }
};

struct Reciprocal : Every<-24, 64> {
  __device__ bool operator()(u64 k, Operands& o) const {
    const float b = o.a = at(k), c = o.b = mirror(k);
    const F2 n = neg_rcp_rn2(F2{b, c});
    return same(rcp_rn(b), __frcp_rn(b)) && same(-n.x, __frcp_rn(b)) && same(-n.y, __frcp_rn(c));
  }
};

struct Root : Every<-100, 100> {
  __device__ bool operator()(u64 k, Operands& o) const {
    const float a = o.a = at(k), c = o.b = mirror(k);
    const F2 n = neg_sqrt_rn2(F2{-a, -c});
    return same(sqrt_rn(a), __fsqrt_rn(a)) && same(-n.x, __fsqrt_rn(a)) && same(-n.y, __fsqrt_rn(c));
  }
};

struct Power : Every<-12, 20> {
  __device__ bool operator()(u64 k, Operands& o) const {
    const float x = o.a = at(k), c = o.b = mirror(k);
    const PairOne one;
    const F2 p = pow73_mid2(F2{x, c}, one);
    return same(pow73_mid(x), rb_pow73f(x)) && same(p.x, rb_pow73f(x)) && same(p.y, rb_pow73f(c));
  }
};

struct OverG {  // every x of [2^-99, the largest float]
  static u64 count() { return 0x7f800000ull - pow2_bits(-99); }
  __device__ bool operator()(u64 k, Operands& o) const {
    const float x = o.a = flt(pow2_bits(-99) + (unsigned)k);
    return same(rb_div_g_mid(x), __fdiv_rn(x, kG));
  }
};

// |a| in [2^-60, 2^60], b in [2^-24, 2^64]: random mantissas, and quotients next to the
// midpoint of two floats, where a wrong last step shows.
struct Quotient {
  __host__ __device__ static constexpr Pairs range() { return Pairs{-60, 60, -24, 64, 1ull << 14}; }
  static u64 count() { return range().count() + 3; }
  __device__ bool operator()(u64 k, Operands& o) const {
    const u64 ends = range().count();
    int ea = 60, eb = 64;
    u64 r = 0;
    float a = 0x1p60f, b = k == ends ? 0x1p-24f : 0x1p64f;
    if (k == ends + 1) a = 0x1p-60f;
    if (k < ends) {
      range().at(k, ea, eb, r);
      a = in_binade(ea, (unsigned)(r >> 32));
      b = in_binade(eb, (unsigned)r);
      if (r >> 63) {
        const float q = in_binade(ea - eb, (unsigned)(r >> 32));  // ea - eb >= -124
        const float near_mid = (float)(((double)q + ldexp(1.0, ea - eb - 24)) * (double)b);
        if (near_mid >= 0x1p-60f && near_mid <= 0x1p60f) a = near_mid;
      }
      if (r >> 62 & 1) a = -a;
      if ((k & 1023) == 0) a = 0.0f;
      if ((k & 1023) == 1) a = -0.0f;
    }
    o.a = a;
    o.b = b;
    const float want = __fdiv_rn(a, b), y = __frcp_rn(b);
    const F2 p = div_rn_by2(F2{a, -a}, F2{b, b}, F2{-y, -y});
    return same(div_rn(a, b), want) && same(div_rn_by(a, b, y), want) && same(p.x, want) && same(p.y, -want) &&
           div_rn_small_ok(a);
  }
};

// Manning's denominator 1 + f / p for any f in [0, 2^40] (zero and subnormals among them)
// and p in [2^-24, 2^45], the powers of depths in [H_DRY, 2^19].
struct Denominator {
  __host__ __device__ static constexpr Pairs range() { return Pairs{-127, 40, -24, 45, 1ull << 14}; }
  static u64 count() { return range().count(); }
  __device__ bool operator()(u64 k, Operands& o) const {
    int ef, ep;
    u64 r;
    range().at(k, ef, ep, r);
    const float f = o.a = in_binade(ef, (k & 255) == 0 ? 0u : (unsigned)(r >> 32)), p = o.b = in_binade(ep, (unsigned)r);
    const float want = 1.0f + __fdiv_rn(f, p);
    const F2 q = div_rn_by2(F2{f, f}, F2{p, p}, neg_rcp_rn2(F2{p, p}));
    return same(1.0f + div_rn(f, p), want) && same(1.0f + q.x, want) && same(1.0f + q.y, want);
  }
};

// manning_divide against the general expression: depths from H_DRY to the largest float and
// infinity, discharges and numerators of any bits, ordinary and zero roughness.
struct Manning {
  static u64 count() { return 1ull << 28; }
  __device__ bool operator()(u64 k, Operands& o) const {
    const u64 r = mix(k), s = mix(r), t = mix(s);
    float h = flt((unsigned)r & 0x7fffffffu);
    if ((k & 3) != 0) h = in_binade((int)(t % 30) - 10, (unsigned)r);  // 2^-10 .. 2^20
    if (!(h >= kHDry)) h = kHDry;
    float q = flt((unsigned)s), num = flt((unsigned)(s >> 32));
    if ((k & 7) > 1) q = in_binade((int)(t >> 8 & 31) - 24, (unsigned)s);
    if ((k & 7) > 2) num = (s >> 63 ? -1.0f : 1.0f) * in_binade((int)(t >> 16 & 63) - 56, (unsigned)(s >> 32));
    const float n = (t >> 24 & 15) == 0 ? 0.0f : (float)(t >> 32 & 1023) * 0.0005f;
    const float dt = in_binade((int)(t >> 44 & 15) - 8, (unsigned)t);
    o.a = num;
    o.b = h;
    const float f = kG * dt * n * n * fabsf(q);
    return same(manning_divide(num, q, h, n, kG, dt), manning_divide_any(num, f, h));
  }
};

// face_slope against the division: surface differences of any bits, any normal cell size.
struct Slope {
  static u64 count() { return 1ull << 28; }
  __device__ bool operator()(u64 k, Operands& o) const {
    const u64 r = mix(k);
    const int e = (k & 1) ? (int)(r >> 56) % 253 - 126 : (int)(r >> 56) % 44 - 22;
    const float de = o.a = flt((unsigned)r), dx = o.b = in_binade(e, (unsigned)(r >> 32));
    return same(face_slope(de, dx, slope_rcp(dx)), __fdiv_rn(de, dx));
  }
};

// Depths, velocities and momenta as states hold them and beyond: zeros, the dry limit,
// ordinary values, and any bits (subnormals, infinities, not a number).
__device__ __forceinline__ float some_depth(u64 r) {
  const unsigned m = (unsigned)(r >> 32);
  switch (r & 15) {
    case 0: return 0.0f;
    case 1: return flt(bits(kHDry) - 2 + (m & 3));  // either side of the dry limit
    case 2: return flt(m & 0x7fffffffu);
    case 3: return flt(m);
    case 4: return in_binade((int)(r >> 8) % 24 + 10, m);  // 2^10 .. 2^33
    default: return in_binade((int)((r >> 8) % 16) - 10, m);  // 2^-10 .. 2^5
  }
}
__device__ __forceinline__ float some_speed(u64 r) {
  const unsigned m = (unsigned)(r >> 32), sign = m & 0x80000000u;
  switch (r & 15) {
    case 0: return flt(sign);
    case 1: return flt(m);
    case 2: return flt(sign | bits(in_binade((int)((r >> 8) % 120) - 60, m)));
    default: return flt(sign | bits(in_binade((int)((r >> 8) % 20) - 16, m)));  // 2^-16 .. 2^3
  }
}

// The Riemann solve, guarded scalar and packed, against the general form. Half of the faces
// run close to critical (a wave speed near zero) or nearly at rest with equal sides.
struct Riemann {
  static u64 count() { return 1ull << 28; }
  struct Face {
    float hl, ul, vl, hr, ur, vr;
  };
  __device__ static Face face(u64 r) {
    const u64 a = mix(r), b = mix(a), c = mix(b), d = mix(c), e = mix(d), g = mix(e);
    Face f{some_depth(a), some_speed(b), some_speed(c), some_depth(d), some_speed(e), some_speed(g)};
    if (r & 1) {
      if (r & 2) f.hr = f.hl;
      if (r & 4) f.ur = f.ul;
      const int off = (int)(g >> 40 & 7) - 3;
      if ((r & 24) == 8) f.ul = flt(bits(sqrtf(kG * fmaxf(f.hl, 0.0f))) + off);
      if ((r & 24) == 16) f.ur = -flt(bits(sqrtf(kG * fmaxf(f.hr, 0.0f))) + off);
    }
    return f;
  }
  __device__ static bool equal(const Face& f, float f0, float f1, float f2) {
    float w0, w1, w2;
    hllc_flux_any(f.hl, f.ul, f.vl, f.hr, f.ur, f.vr, w0, w1, w2);
    return same(f0, w0) && same(f1, w1) && same(f2, w2);
  }
  __device__ bool operator()(u64 k, Operands& o) const {
    const Face f = face(mix(2 * k)), h = face(mix(2 * k + 1));
    o = Operands{f.hl, f.hr};
    float f0, f1, f2;
    hllc_flux(f.hl, f.ul, f.vl, f.hr, f.ur, f.vr, f0, f1, f2);
    F2 p0, p1, p2;
    bool odd = false;
    hllc_near2(F2{f.hl, h.hl}, F2{f.ul, h.ul}, F2{f.vl, h.vl}, F2{f.hr, h.hr}, F2{f.ur, h.ur}, F2{f.vr, h.vr}, p0, p1,
               p2, odd);
    return equal(f, f0, f1, f2) && (odd || (equal(f, p0.x, p1.x, p2.x) && equal(h, p0.y, p1.y, p2.y)));
  }
};

// A cell's primitives, friction and wave speed, guarded, against the general forms.
struct CellValues {
  static u64 count() { return 1ull << 28; }
  __device__ bool operator()(u64 k, Operands& o) const {
    const u64 a = mix(k), b = mix(a), c = mix(b), d = mix(c);
    const float h = some_depth(a), hu = some_speed(b), hv = (c & 0x300) == 0 ? hu : some_speed(c);
    o = Operands{h, hu};
    float u, v, wu, wv;
    primitives(h, hu, hv, u, v);
    primitives_any(h, hu, hv, wu, wv);
    const bool wet = h > kHDry;
    const float n = (d & 15) == 0 ? 0.0f : (d & 15) == 1 ? flt((unsigned)(d >> 32)) : (float)(d >> 8 & 1023) * 0.0005f;
    const float gdt = kG * in_binade((int)(d >> 20 & 15) - 8, (unsigned)(d >> 32));
    float qu = hu, qv = hv, gu = hu, gv = hv;
    hllc_friction<false>(h, wet, gdt, n, qu, qv);
    friction_any(h, wet, gdt, n, gu, gv);
    return same(u, wu) && same(v, wv) && same(qu, gu) && same(qv, gv) &&
           same(wave_speed<false>(h, hu, hv), wave_speed_any(h, hu, hv));
  }
};
#else
// The bounds are those of the units' documentation (reciprocal: 1 ulp; square root: 2^-23;
// logarithm: 2^-22 of max(1, |result|); exponential: 2 ulp of the rounded result) and of
// the roundings between them, with 2^-40 for the reference's own.
constexpr double kSlack = 1.0 + 0x1p-40;

struct Quotient {
  __host__ __device__ static constexpr Pairs range() { return Pairs{-60, 60, -60, 60, 1ull << 14}; }
  static u64 count() { return range().count(); }
  __device__ bool operator()(u64 k, Operands& o) const {
    int ea, eb;
    u64 r;
    range().at(k, ea, eb, r);
    const float a = o.a = in_binade(ea, (unsigned)(r >> 32)), b = o.b = in_binade(eb, (unsigned)r);
    const double got = (double)__fmul_rn(a, rcp_near(b)), want = (double)a / (double)b;
    return fabs(got - want) <= 0x1p-22 * kSlack * want;
  }
};

struct Root {  // every normal float
  static u64 count() { return 0x7f800000ull - 0x00800000ull; }
  __device__ bool operator()(u64 k, Operands& o) const {
    const float a = o.a = flt(0x00800000u + (unsigned)k);
    const double want = sqrt((double)a);
    return fabs((double)sqrt_near(a) - want) <= 0x1p-23 * kSlack * want;
  }
};

struct Power {  // every depth of [H_DRY, 2^20]
  static u64 count() { return (u64)pow2_bits(20) - 0x3a83126full + 1; }
  __device__ bool operator()(u64 k, Operands& o) const {
    const float h = o.a = flt(0x3a83126fu + (unsigned)k);
    const double p = (double)2.33333325f, want = pow((double)h, p), l = fabs(log2((double)h));
    const double bound = 0.6931471805599453 * (p * 0x1p-22 * fmax(1.0, l) + 0x1p-24 * p * l) + 0x1p-22 + 0x1p-24;
    const double got = (double)pow73_near(h);
    // exp(bound) - 1 for the exponential's part of it
    return fabs(got - want) <= (bound + bound * bound) * kSlack * want && got > 0x1p-24;
  }
};
#endif

template <class Check>
__global__ void __launch_bounds__(256) sweep_kernel(u64 n, u64* bad, Operands* first) {
  const Check check;
  for (u64 k = (u64)blockIdx.x * 256 + threadIdx.x; k < n; k += (u64)gridDim.x * 256) {
    Operands o{0.0f, 0.0f};
    if (!check(k, o) && atomicAdd(bad, 1ull) == 0) *first = o;
  }
}

template <class Check>
int sweep(u64* tried, u64* bad, float* first) {
  struct Result {
    u64 bad;
    Operands first;
  } host{}, *dev = nullptr;
  cudaError_t e = cudaMalloc(&dev, sizeof host);
  if (e != cudaSuccess) return (int)e;
  e = cudaMemset(dev, 0, sizeof host);
  if (e == cudaSuccess) {
    sweep_kernel<Check><<<148 * 8, 256>>>(Check::count(), &dev->bad, &dev->first);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(&host, dev, sizeof host, cudaMemcpyDeviceToHost);
  cudaFree(dev);
  *tried = Check::count();
  *bad = host.bad;
  first[0] = host.first.a;
  first[1] = host.first.b;
  return (int)e;
}

#define RB_SWEEP(name, Check) \
  extern "C" int sweep_##name(u64* tried, u64* bad, float* first) { return sweep<Check>(tried, bad, first); }
RB_SWEEP(quotient, Quotient)
RB_SWEEP(root, Root)
RB_SWEEP(power, Power)
#if !defined(RB_FAST_MATH)
RB_SWEEP(reciprocal, Reciprocal)
RB_SWEEP(over_g, OverG)
RB_SWEEP(denominator, Denominator)
RB_SWEEP(manning, Manning)
RB_SWEEP(slope, Slope)
RB_SWEEP(riemann, Riemann)
RB_SWEEP(cell_values, CellValues)
#endif

RB_ARITH_END
}  // namespace rb
