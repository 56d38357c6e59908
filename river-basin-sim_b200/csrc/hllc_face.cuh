// hllc_face.cuh -- the HLLC step's arithmetic of a face and a cell: the Riemann solve, the
// primitives, friction and the wave speed.
//
// Included by hllc_step.cu inside its arithmetic namespace, after pair.cuh and
// warp_stream.cuh.
#pragma once

#if !defined(RB_FAST_MATH)
// hllc.py:191-256 _hllc: (mass, normal momentum, transverse momentum) flux.
__device__ __forceinline__ void hllc_flux_any(float hl, float ul, float vtl, float hr, float ur, float vtr, float& f0,
                                          float& f1, float& f2) {
  const float g = kG;
  const float cl = sqrtf(g * rmax(hl, 0.0f));
  const float cr = sqrtf(g * rmax(hr, 0.0f));
  const bool dry_l = hl <= kHDry, dry_r = hr <= kHDry;
  if (dry_l && dry_r) {
    f0 = 0.0f;
    f1 = 0.0f;
    f2 = 0.0f;
    return;
  }
  float sl, sr;
  if (dry_l) {
    sl = ur - 2.0f * cr;
    sr = ur + cr;
  } else if (dry_r) {
    sl = ul - cl;
    sr = ul + 2.0f * cl;
  } else {
    const float hs = 0.5f * (cl + cr) + 0.25f * (ul - ur);
    const float h_star = rmax(div_g(hs * hs), 0.0f);  // hs * hs / g
    const float c_star = sqrtf(g * h_star);
    const float u_star = 0.5f * (ul + ur) + cl - cr;
    sl = rmin(ul - cl, u_star - c_star);
    sr = rmax(ur + cr, u_star + c_star);
  }
  const float fh_l = hl * ul;
  const float fmn_l = hl * ul * ul + 0.5f * g * hl * hl;
  const float fh_r = hr * ur;
  const float fmn_r = hr * ur * ur + 0.5f * g * hr * hr;
  float fh, fmn;
  if (sl >= 0.0f) {
    fh = fh_l;
    fmn = fmn_l;
  } else if (sr <= 0.0f) {
    fh = fh_r;
    fmn = fmn_r;
  } else {
    const float inv = 1.0f / (sr - sl);
    fh = (sr * fh_l - sl * fh_r + sl * sr * (hr - hl)) * inv;
    fmn = (sr * fmn_l - sl * fmn_r + sl * sr * (hr * ur - hl * ul)) * inv;
  }
  // The contact speed s_star is read only through s_star >= 0 (hllc.py:231-238), so
  // its sign is decided without the division (quotient_nonneg).
  const float den_s = hr * (ur - sr) - hl * (ul - sl);
  const bool star_nonneg = fabsf(den_s) > 1.0e-12f
                               ? quotient_nonneg(sl * hr * (ur - sr) - sr * hl * (ul - sl), den_s)
                               : 0.5f * (ul + ur) >= 0.0f;
  const float vt = star_nonneg ? vtl : vtr;
  f0 = fh;
  f1 = fmn;
  f2 = fh * vt;
}

// hllc.py:262-282 _primitives: u = hu / h and v = hv / h on a wet cell, 0 on a dry
// one. Still water (hu = hv = 0) is common, and its quotients are the zero momenta
// themselves, so such cells branch around both divisions (a zero dividend would take
// the division's slow path); a cell with one zero momentum divides 1 in its place.
__device__ __forceinline__ void primitives_any(float h, float hu, float hv, float& u, float& v) {
  const bool wet = h > kHDry;
  u = wet ? hu : 0.0f;
  v = wet ? hv : 0.0f;
  if (wet && !(hu == 0.0f && hv == 0.0f)) {
    const float qu = div_in_branch(opaque(hu == 0.0f ? 1.0f : hu), h);
    const float qv = div_in_branch(opaque(hv == 0.0f ? 1.0f : hv), h);
    if (hu != 0.0f) u = qu;
    if (hv != 0.0f) v = qv;
  }
}

// Manning friction on the new momenta of a wet cell (hllc.py:912-939): the numerator
// g dt n^2 |q| is zero, and the denominator exactly 1 so hu and hv stand as they are,
// whenever n = 0 with a finite |q|^2 or the water is still with a finite g dt n^2;
// neither the square root nor the power is needed then.
__device__ __forceinline__ void friction_any(float hh, bool wet, float gdt, float n, float& hu, float& hv) {
  const float m2 = hu * hu + hv * hv;
  const float k = gdt * n * n;
  if (wet && !((k == 0.0f && m2 <= FLT_MAX) || (m2 == 0.0f && k <= FLT_MAX))) {
    const float f = k * sqrtf(m2);
    if (!(f == 0.0f)) {
      const float denom = 1.0f + f / pow73(hh);
      hu = div_pos(hu, denom);
      hv = div_pos(hv, denom);
    }
  }
}

// max(|u|, |v|) + sqrt(g h) of a cell (hllc.py:948-966 _reduce_wavespeed).
__device__ __forceinline__ float wave_speed_any(float hh, float hu, float hv) {
  const float cw = sqrtf(kG * rmax(hh, 0.0f));
  const bool wet = hh > kHDry;
  return wet ? rmax(div_if(wet, fabsf(hu), hh), div_if(wet, fabsf(hv), hh)) + cw : cw;
}

#endif  // !RB_FAST_MATH

// The cell and face arithmetic as the kernels evaluate it. Exact build: the values of the
// `_any` functions above without branches, by correctly rounded divisions and square roots
// inside a safe range (rcp_rn, div_rn, sqrt_rn); `odd` is set where an operand leaves it,
// and the caller redoes those with the `_any` function. VOTE: every lane of the warp calls
// (the row-streaming kernels), so a warp can skip what none of its lanes needs.
#if defined(RB_FAST_MATH)
// Fast arithmetic: the approximate units in their flush-to-zero forms, the star celerity as
// |hs| (sqrt(g max(hs^2 / g, 0))), the three HLL cases in one formula (with the wave speeds
// clamped to sl <= 0 <= sr the HLL flux is the left one when sl >= 0 and the right one when
// sr <= 0, to rounding; sl < sr whenever one side is wet), the contact speed's sign from a
// product, one reciprocal per cell.
__device__ __forceinline__ void primitives_near(float h, float hu, float hv, float& u, float& v, bool&) {
  const bool wet = h > kHDry;
  const float r = rcp_near(wet ? h : 1.0f);
  u = wet ? hu * r : 0.0f;
  v = wet ? hv * r : 0.0f;
}

__device__ __forceinline__ void hllc_near(float hl, float ul, float vtl, float hr, float ur, float vtr, float& f0,
                                          float& f1, float& f2, bool&) {
  const float g = kG;
  const float cl = sqrt_near(g * fmaxf(hl, 0.0f)), cr = sqrt_near(g * fmaxf(hr, 0.0f));
  const bool dry_l = hl <= kHDry, dry_r = hr <= kHDry;
  const float c_star = fabsf(0.5f * (cl + cr) + 0.25f * (ul - ur));
  const float u_star = 0.5f * (ul + ur) + cl - cr;
  float sl = fminf(ul - cl, u_star - c_star), sr = fmaxf(ur + cr, u_star + c_star);
  if (dry_r) sl = ul - cl, sr = ul + 2.0f * cl;
  if (dry_l) sl = ur - 2.0f * cr, sr = ur + cr;
  const float fh_l = hl * ul, fmn_l = hl * ul * ul + 0.5f * g * hl * hl;
  const float fh_r = hr * ur, fmn_r = hr * ur * ur + 0.5f * g * hr * hr;
  const float a = fminf(sl, 0.0f), b = fmaxf(sr, 0.0f);
  const float inv = rcp_near(fmaxf(b - a, 1.0e-30f));
  const float fh = (b * fh_l - a * fh_r + a * b * (hr - hl)) * inv;
  const float fmn = (b * fmn_l - a * fmn_r + a * b * (hr * ur - hl * ul)) * inv;
  const float den_s = hr * (ur - sr) - hl * (ul - sl);
  const bool star_nonneg =
      fabsf(den_s) > 1.0e-12f ? (sl * hr * (ur - sr) - sr * hl * (ul - sl)) * den_s >= 0.0f : ul + ur >= 0.0f;
  const bool none = dry_l && dry_r;
  f0 = none ? 0.0f : fh;
  f1 = none ? 0.0f : fmn;
  f2 = none ? 0.0f : fh * (star_nonneg ? vtl : vtr);
}

// hllc_near for the two faces that are the halves of its operands (to rounding).
__device__ __forceinline__ void hllc_near2(F2 hl, F2 ul, F2 vtl, F2 hr, F2 ur, F2 vtr, F2& f0, F2& f1, F2& f2, bool&) {
  const float g = kG;
  const F2 gl = g * F2{fmaxf(hl.x, 0.0f), fmaxf(hl.y, 0.0f)}, gr = g * F2{fmaxf(hr.x, 0.0f), fmaxf(hr.y, 0.0f)};
  const F2 cl{sqrt_near(gl.x), sqrt_near(gl.y)}, cr{sqrt_near(gr.x), sqrt_near(gr.y)};
  const bool dlx = hl.x <= kHDry, dly = hl.y <= kHDry, drx = hr.x <= kHDry, dry = hr.y <= kHDry;
  const F2 hs = fma2(both(0.25f), ul - ur, 0.5f * (cl + cr)), usum = ul + ur;
  const F2 c_star{fabsf(hs.x), fabsf(hs.y)}, u_star = fma2(both(0.5f), usum, cl - cr);
  const F2 ulm = ul - cl, urp = ur + cr, sm = u_star - c_star, sp = u_star + c_star;
  const F2 ul2 = fma2(both(2.0f), cl, ul), ur2 = fma2(both(-2.0f), cr, ur);
  F2 sl{fminf(ulm.x, sm.x), fminf(ulm.y, sm.y)}, sr{fmaxf(urp.x, sp.x), fmaxf(urp.y, sp.y)};
  if (drx) sl.x = ulm.x, sr.x = ul2.x;
  if (dry) sl.y = ulm.y, sr.y = ul2.y;
  if (dlx) sl.x = ur2.x, sr.x = urp.x;
  if (dly) sl.y = ur2.y, sr.y = urp.y;
  const F2 fh_l = hl * ul, fmn_l = fma2(fh_l, ul, 0.5f * g * hl * hl);
  const F2 fh_r = hr * ur, fmn_r = fma2(fh_r, ur, 0.5f * g * hr * hr);
  // -min(sl, 0) and max(sr, 0)
  const F2 a{fmaxf(-sl.x, 0.0f), fmaxf(-sl.y, 0.0f)}, b{fmaxf(sr.x, 0.0f), fmaxf(sr.y, 0.0f)};
  const F2 gap = a + b, ab = a * b;
  const F2 inv{rcp_near(fmaxf(gap.x, 1.0e-30f)), rcp_near(fmaxf(gap.y, 1.0e-30f))};
  const F2 fh = fma2(b, fh_l, fma2(a, fh_r, ab * (hl - hr))) * inv;
  const F2 fmn = fma2(b, fmn_l, fma2(a, fmn_r, ab * (fh_l - fh_r))) * inv;
  const F2 mr = hr * (ur - sr), ml = hl * (sl - ul);
  const F2 den_s = mr + ml, num_s = fma2(sl, mr, sr * ml), sgn = num_s * den_s;
  const bool tx = fabsf(den_s.x) > 1.0e-12f ? sgn.x >= 0.0f : usum.x >= 0.0f;
  const bool ty = fabsf(den_s.y) > 1.0e-12f ? sgn.y >= 0.0f : usum.y >= 0.0f;
  const bool nx = dlx && drx, ny = dly && dry;
  const F2 ft = fh * F2{tx ? vtl.x : vtr.x, ty ? vtl.y : vtr.y};
  f0 = F2{nx ? 0.0f : fh.x, ny ? 0.0f : fh.y};
  f1 = F2{nx ? 0.0f : fmn.x, ny ? 0.0f : fmn.y};
  f2 = F2{nx ? 0.0f : ft.x, ny ? 0.0f : ft.y};
}

template <bool VOTE>
__device__ __forceinline__ void hllc_friction(float hh, bool wet, float gdt, float n, float& hu, float& hv) {
  const float f = gdt * n * n * sqrt_near(hu * hu + hv * hv);
  const float rd = rcp_near(1.0f + f * rcp_near(pow73_near(hh)));
  if (wet) hu *= rd, hv *= rd;
}

template <bool VOTE>
__device__ __forceinline__ float wave_speed(float hh, float hu, float hv) {
  const float cw = sqrt_near(kG * fmaxf(hh, 0.0f));
  const bool wet = hh > kHDry;
  return wet ? rmax(fabsf(hu), fabsf(hv)) * rcp_near(wet ? hh : 1.0f) + cw : cw;
}

__device__ __forceinline__ void primitives(float h, float hu, float hv, float& u, float& v) {
  bool odd;
  primitives_near(h, hu, hv, u, v, odd);
}
__device__ __forceinline__ void hllc_flux(float hl, float ul, float vtl, float hr, float ur, float vtr, float& f0,
                                          float& f1, float& f2) {
  bool odd;
  hllc_near(hl, ul, vtl, hr, ur, vtr, f0, f1, f2, odd);
}
#else
__device__ __forceinline__ void primitives_near(float h, float hu, float hv, float& u, float& v, bool& odd) {
  const bool wet = h > kHDry;
  const float hs = wet ? h : 1.0f, y = rcp_rn(hs);
  const float qu = div_rn_by(hu, hs, y), qv = div_rn_by(hv, hs, y);
  u = wet ? qu : 0.0f;
  v = wet ? qv : 0.0f;
  const float m = fmaxf(fabsf(hu), fabsf(hv));
  odd |= wet & !(div_rn_small_ok(hu) & div_rn_small_ok(hv) & (h <= 0x1p24f) & (m <= 0x1p60f));
}

__device__ __forceinline__ void hllc_near(float hl, float ul, float vtl, float hr, float ur, float vtr, float& f0,
                                          float& f1, float& f2, bool& odd) {
  const float g = kG;
  const bool dry_l = hl <= kHDry, dry_r = hr <= kHDry, none = dry_l & dry_r;
  // a dry side's celerity is not used
  const float cl = sqrt_rn(g * (dry_l ? 1.0f : hl)), cr = sqrt_rn(g * (dry_r ? 1.0f : hr));
  const float hs = 0.5f * (cl + cr) + 0.25f * (ul - ur);
  const float hs2 = hs * hs;
  const float c_star = sqrt_rn(g * rb_div_g_mid(hs2));
  const float u_star = 0.5f * (ul + ur) + cl - cr;
  float sl = rmin(ul - cl, u_star - c_star), sr = rmax(ur + cr, u_star + c_star);
  if (dry_r) sl = ul - cl, sr = ul + 2.0f * cl;
  if (dry_l) sl = ur - 2.0f * cr, sr = ur + cr;
  const float fh_l = hl * ul, fmn_l = hl * ul * ul + 0.5f * g * hl * hl;
  const float fh_r = hr * ur, fmn_r = hr * ur * ur + 0.5f * g * hr * hr;
  const float gap = sr - sl, inv = rcp_rn(gap);
  const float fh_m = (sr * fh_l - sl * fh_r + sl * sr * (hr - hl)) * inv;
  const float fmn_m = (sr * fmn_l - sl * fmn_r + sl * sr * (hr * ur - hl * ul)) * inv;
  const float fh = sl >= 0.0f ? fh_l : (sr <= 0.0f ? fh_r : fh_m);
  const float fmn = sl >= 0.0f ? fmn_l : (sr <= 0.0f ? fmn_r : fmn_m);
  // the sign of the contact speed num_s / den_s (quotient_nonneg without its rare cases)
  const float den_s = hr * (ur - sr) - hl * (ul - sl);
  const float num_s = sl * hr * (ur - sr) - sr * hl * (ul - sl);
  const bool have_s = fabsf(den_s) > 1.0e-12f;
  const bool nonneg = have_s ? (num_s == 0.0f) | ((num_s > 0.0f) == (den_s > 0.0f)) : 0.5f * (ul + ur) >= 0.0f;
  const bool sign_ok = !have_s | (num_s == 0.0f) | (fabsf(num_s) > fabsf(den_s) * 0x1p-100f);
  f0 = none ? 0.0f : fh;
  f1 = none ? 0.0f : fmn;
  f2 = none ? 0.0f : fh * (nonneg ? vtl : vtr);
  odd |= !none & !((gap >= 0x1p-20f) & (gap <= 0x1p50f) & (dry_l | dry_r | (hs2 >= 0x1p-99f)) & sign_ok);
}

// hllc_near for the two faces that are the halves of its operands, the same bits. The
// streaming kernel is bound by the instructions it issues (with pairs in 69 to 73 % of its
// cycles), and half of them are adds and multiplies: 745 -> 648 instructions a cell in stage 1
// (2048^2, us per step: lake 290 -> 270, dam break 268 -> 246; fast dam break 190 -> 178).
__device__ __forceinline__ void hllc_near2(F2 hl, F2 ul, F2 vtl, F2 hr, F2 ur, F2 vtr, F2& f0, F2& f1, F2& f2,
                                           bool& odd) {
  const float g = kG;
  const PairOne one;
  const bool dlx = hl.x <= kHDry, dly = hl.y <= kHDry, drx = hr.x <= kHDry, dry = hr.y <= kHDry;
  const bool nx = dlx & drx, ny = dly & dry;
  const F2 ncl = neg_sqrt_rn2(-g * F2{dlx ? 1.0f : hl.x, dly ? 1.0f : hl.y});
  const F2 ncr = neg_sqrt_rn2(-g * F2{drx ? 1.0f : hr.x, dry ? 1.0f : hr.y});
  const F2 usum = 0.5f * (ul + ur);
  const F2 hs = 0.25f * (ul - ur) - 0.5f * (ncl + ncr);
  const F2 hs2 = hs * hs;
  const F2 nc_star = neg_sqrt_rn2(-g * fma2(hs2, both(0x1.a1887ap-4f), 0x1.dcb5p-38f * hs2));
  const F2 u_star = usum - ncl + ncr;
  const F2 ulm = ul + ncl, urp = ur - ncr, sm = u_star + nc_star, sp = u_star - nc_star;
  const F2 ul2 = ul - (ncl + ncl), ur2 = ur + (ncr + ncr);
  F2 sl{rmin(ulm.x, sm.x), rmin(ulm.y, sm.y)}, sr{rmax(urp.x, sp.x), rmax(urp.y, sp.y)};
  if (drx) sl.x = ulm.x, sr.x = ul2.x;
  if (dry) sl.y = ulm.y, sr.y = ul2.y;
  if (dlx) sl.x = ur2.x, sr.x = urp.x;
  if (dly) sl.y = ur2.y, sr.y = urp.y;
  const F2 fh_l = hl * ul, fmn_l = one.add(fh_l * ul, 0.5f * g * hl * hl);
  const F2 fh_r = hr * ur, fmn_r = one.add(fh_r * ur, 0.5f * g * hr * hr);
  const F2 ngap = sl - sr, gap{-ngap.x, -ngap.y};
  F2 y0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0.x) : "f"(gap.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0.y) : "f"(gap.y));
  const F2 inv = fma2(fma2(ngap, y0, both(1.0f)), y0, y0);  // rcp_rn(gap)
  const F2 slsr = sl * sr;
  const F2 fh_m = one.add(one.sub(sr * fh_l, sl * fh_r), slsr * (hr - hl)) * inv;
  const F2 fmn_m = one.add(one.sub(sr * fmn_l, sl * fmn_r), slsr * one.sub(fh_r, fh_l)) * inv;
  const F2 ursr = ur - sr, ulsl = ul - sl;
  const F2 den_s = one.sub(hr * ursr, hl * ulsl);
  const F2 num_s = one.sub(sl * hr * ursr, sr * hl * ulsl);
  auto finish = [&](float sl, float sr, float fh_l, float fh_r, float fh_m, float fmn_l, float fmn_r, float fmn_m,
                    float den_s, float num_s, float usum, float vtl, float vtr, bool none, float& f0, float& f1,
                    float& f2) {
    const float fh = sl >= 0.0f ? fh_l : (sr <= 0.0f ? fh_r : fh_m);
    const float fmn = sl >= 0.0f ? fmn_l : (sr <= 0.0f ? fmn_r : fmn_m);
    const bool have_s = fabsf(den_s) > 1.0e-12f;
    const bool nonneg = have_s ? (num_s == 0.0f) | ((num_s > 0.0f) == (den_s > 0.0f)) : usum >= 0.0f;
    f0 = none ? 0.0f : fh;
    f1 = none ? 0.0f : fmn;
    f2 = none ? 0.0f : fh * (nonneg ? vtl : vtr);
    return !have_s | (num_s == 0.0f) | (fabsf(num_s) > fabsf(den_s) * 0x1p-100f);
  };
  const bool okx = finish(sl.x, sr.x, fh_l.x, fh_r.x, fh_m.x, fmn_l.x, fmn_r.x, fmn_m.x, den_s.x, num_s.x, usum.x,
                          vtl.x, vtr.x, nx, f0.x, f1.x, f2.x);
  const bool oky = finish(sl.y, sr.y, fh_l.y, fh_r.y, fh_m.y, fmn_l.y, fmn_r.y, fmn_m.y, den_s.y, num_s.y, usum.y,
                          vtl.y, vtr.y, ny, f0.y, f1.y, f2.y);
  odd |= !nx & !((gap.x >= 0x1p-20f) & (gap.x <= 0x1p50f) & (dlx | drx | (hs2.x >= 0x1p-99f)) & okx);
  odd |= !ny & !((gap.y >= 0x1p-20f) & (gap.y <= 0x1p50f) & (dly | dry | (hs2.y >= 0x1p-99f)) & oky);
}

template <bool VOTE>
__device__ __forceinline__ void hllc_friction(float hh, bool wet, float gdt, float n, float& hu, float& hv) {
  const float m2 = hu * hu + hv * hv, k = gdt * n * n;
  const bool need = wet & !(((k == 0.0f) & (m2 <= FLT_MAX)) | ((m2 == 0.0f) & (k <= FLT_MAX)));
  if (!any_lane<VOTE>(need)) return;
  const float f = k * sqrt_rn(need ? m2 : 1.0f);
  const float den = 1.0f + div_rn(f, pow73_mid(need ? hh : 1.0f));
  const float y = rcp_rn(den);
  const float qu = div_rn_by(hu, den, y), qv = div_rn_by(hv, den, y);
  const bool ok = (m2 >= 0x1p-100f) & (m2 <= 0x1p100f) & (hh <= 0x1p19f) & (f <= 0x1p40f) & (den <= 0x1p20f) &
                  div_rn_small_ok(hu) & div_rn_small_ok(hv);
  if (any_lane<VOTE>(need & !ok))
    friction_any(hh, wet, gdt, n, hu, hv);
  else if (need)
    hu = qu, hv = qv;
}

// max(|u|, |v|) + sqrt(g h) of a cell (hllc.py:948-966 _reduce_wavespeed). The larger
// quotient is the larger dividend's: rounding is monotonic.
template <bool VOTE>
__device__ __forceinline__ float wave_speed(float hh, float hu, float hv) {
  const bool wet = hh > kHDry;
  const float a = rmax(fabsf(hu), fabsf(hv)), hs = wet ? hh : 1.0f;
  const bool ok = !wet | ((hh <= 0x1p24f) & (a <= 0x1p60f) & div_rn_small_ok(a));
  if (any_lane<VOTE>(!ok | ((hh > 0.0f) & !(hh >= 0x1p-100f)))) return wave_speed_any(hh, hu, hv);
  const float cw = hh > 0.0f ? sqrt_rn(kG * hh) : 0.0f;
  return wet ? div_rn(a, hs) + cw : cw;
}

__device__ __forceinline__ void primitives(float h, float hu, float hv, float& u, float& v) {
  bool odd = false;
  primitives_near(h, hu, hv, u, v, odd);
  if (odd) primitives_any(h, hu, hv, u, v);
}
__device__ __forceinline__ void hllc_flux(float hl, float ul, float vtl, float hr, float ur, float vtr, float& f0,
                                          float& f1, float& f2) {
  bool odd = false;
  hllc_near(hl, ul, vtl, hr, ur, vtr, f0, f1, f2, odd);
  if (odd) hllc_flux_any(hl, ul, vtl, hr, ur, vtr, f0, f1, f2);
}
#endif
