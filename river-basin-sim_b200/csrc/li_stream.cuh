// li_stream.cuh -- the local-inertial step as a row-streaming kernel.
//
// Included by li_step.cu inside its arithmetic namespace, after the face helpers.
//
// A warp owns a strip of 32 columns (a cell a lane) and walks down the
// rows of its chunk. Everything a row needs from the rows above is in registers, and
// everything it needs from the cells to its left and right comes by warp shuffle, so
// each face flux, each beta and each update is computed once per strip, with no
// shared memory and no barrier in the loop. Row r enters at iteration r:
//   r    : eta, the unlimited x-faces of row r and the unlimited y-face above it
//   r - 1: its four faces are known now: beta; its x-faces and the y-face above it are
//          limited, integrated (bedload) and stored
//   r - 2: its four limited faces are known now: continuity, sources, sinks, stored
// The outer two columns on either side of a strip and two rows above and below a chunk
// are computed by the neighbouring warps as well and stored by them.
#pragma once

constexpr int kLiHalo = 2;
constexpr int kLiStreamCols = 32 - 2 * kLiHalo;  // columns a strip stores
constexpr int kLiStreamWarps = 24;               // resident warps per SM (at most 80 registers a thread)

// Constants of a step's faces.
struct LiFaceConst {
  float dt, dx, rdx;  // rdx = 1 / dx, rounded once (fast arithmetic: the approximate reciprocal)
  float gdt;          // g * dt
};

// NF unlimited faces of a warp's lanes (local_inertial.py:72-129), each between a low
// cell (west / north, surface el) and a high one (er), with the flow depth h over the
// higher bed, mean roughness n and previous discharge qo; 0 where !on or h < H_DRY.
#if defined(RB_FAST_MATH)
template <int NF>
__device__ __forceinline__ void li_faces(const float (&qo)[NF], const float (&el)[NF], const float (&er)[NF],
                                         const float (&h)[NF], const float (&n)[NF], const bool (&on)[NF],
                                         const LiFaceConst& c, float (&q)[NF]) {
#pragma unroll
  for (int i = 0; i < NF; i++) {
    const float slope = (er[i] - el[i]) * c.rdx;
    const float num = qo[i] - kG * h[i] * c.dt * slope;
    const float v = manning_divide(num, qo[i], h[i], n[i], kG, c.dt);
    q[i] = !on[i] || h[i] < kHDry ? 0.0f : v;
  }
}
#else
// Exact arithmetic, without a branch per face: the divisions are div_rn (rb_common.cuh)
// on operands inside its range, and a warp with a face outside it takes the reference's
// expressions face by face. A friction numerator f below 2^-60 cannot lift the
// denominator off 1 (h^(7/3) > 2^-24), so the discharge is the numerator itself; a warp
// with no larger one skips the powers. The x-face and the y-face of a row are the halves
// of packed pairs (pair.cuh): 97.9 -> 91.6 us per 2048^2 step.
template <int NF>
__device__ __forceinline__ void li_faces(const float (&qo)[NF], const float (&el)[NF], const float (&er)[NF],
                                         const float (&h)[NF], const float (&n)[NF], const bool (&on)[NF],
                                         const LiFaceConst& c, float (&q)[NF]) {
  static_assert(NF == 2, "the faces are the halves of packed pairs");
  const PairOne one;
  const F2 ho{h[0], h[1]}, no{n[0], n[1]}, qp{qo[0], qo[1]};
  const F2 de = F2{er[0], er[1]} - F2{el[0], el[1]};
  const F2 num = one.sub(qp, kG * ho * both(c.dt) * div_rn_by2(de, both(c.dx), both(-c.rdx)));
  const F2 f = c.gdt * no * no * F2{fabsf(qo[0]), fabsf(qo[1])};
  bool wet[NF], need = false, odd = c.rdx == 0.0f;
  auto check = [&](bool on, float h, float de, float num, float f, bool& wet, float& q) {
    wet = on & !(h < kHDry);
    const bool small = div_rn_small_ok(de) & div_rn_small_ok(num);
    const bool large = !(fmaxf(fabsf(de), fabsf(num)) > 0x1p60f) & (h <= 0x1p19f) & (f <= 0x1p40f);
    odd |= wet & !(small & large);
    need |= wet & (f >= 0x1p-60f);
    q = wet ? num : 0.0f;
  };
  check(on[0], h[0], de.x, num.x, f.x, wet[0], q[0]);
  check(on[1], h[1], de.y, num.y, f.y, wet[1], q[1]);
  if (__any_sync(kFullWarp, need)) {
    const F2 p = pow73_mid2(F2{wet[0] ? h[0] : 1.0f, wet[1] ? h[1] : 1.0f}, one);
    const F2 ratio = div_rn_by2(f, p, neg_rcp_rn2(p));
    const F2 den = both(1.0f) + ratio;
    odd |= (wet[0] & !(den.x <= 0x1p20f)) | (wet[1] & !(den.y <= 0x1p20f));
    const F2 v = div_rn_by2(num, den, neg_rcp_rn2(den));
    q[0] = wet[0] ? v.x : 0.0f;
    q[1] = wet[1] ? v.y : 0.0f;
  }
  if (__any_sync(kFullWarp, odd)) {
#pragma unroll 1
    for (int i = 0; i < NF; i++) {
      float qi = 0.0f, o = 0.0f, l = 0.0f, r = 0.0f, hh = 1.0f, nn = 0.0f;
      bool w = false;
#pragma unroll
      for (int j = 0; j < NF; j++) {
        if (j == i) o = qo[j], l = el[j], r = er[j], hh = h[j], nn = n[j], w = wet[j];
      }
      if (w)
        qi = manning_divide_any(o - kG * hh * c.dt * div_pos(r - l, c.dx), c.gdt * nn * nn * fabsf(o), hh);
#pragma unroll
      for (int j = 0; j < NF; j++) {
        if (j == i) q[j] = qi;
      }
    }
  }
}
#endif

__device__ __forceinline__ LiFaceConst li_face_const(float dt, float dx) {
  LiFaceConst c;
  c.dt = dt;
  c.dx = dx;
  c.rdx = slope_rcp(dx);
  c.gdt = kG * dt;
  return c;
}

// Per-cell sources of a step: none beyond a uniform rain added plainly, the compensated
// uniform rain, or whatever the pointers say (rain field, infiltration).
enum { kLiSrcNone = 0, kLiSrcComp = 1, kLiSrcAny = 2 };

// A warp's staging area: the row in use and the one on its way, each lane's word of
// every array its iteration reads. Two rows measured the same as four without bedload
// (0.170 against 0.174 ms per 4096^2 fast step) and better with it (1.19 against 1.52 ms
// on the 8192^2 reach: four rows of 13 arrays leave the L1 cache too little).
template <int SED, int SRC>
struct LiRing {
  static constexpr int kComp = 5, kRain = kComp + (SRC != kLiSrcNone), kInfil = kRain + (SRC == kLiSrcAny);
  static constexpr int kD50 = kInfil + (SRC == kLiSrcAny);
  static constexpr int N = kD50 + (SED != 0 ? 5 : 0);
  static constexpr int kStage = (N <= 8 ? 8 : 16) * 32;  // floats a row, a power of two
  alignas(16) float row[2 * kStage];
};

// Rows [i0, i1) of the strip whose first column (lane 0) is c0. EDGE: the strip or its
// halo may reach a domain edge (bounds checks and sinks); the other instantiation is for
// strips whose every staged cell and face is an inner one. Element offsets are 32-bit,
// relative to the row two above the chunk (the launcher keeps a chunk below 2^31).
template <int SED, int SRC, bool EDGE>
__device__ __forceinline__ void li_stream_strip(const LiParams& p, const LiStepScalars& s, int c0, int i0, int i1,
                                                LiRing<SED, SRC>& ring, double& loss, float& hmax, bool& bad) {
  using Ring = LiRing<SED, SRC>;
  const int lane = threadIdx.x & 31;
  const int ny = p.ny, nx = p.nx;
  const float dt = s.dt, dx = p.dx32;
  const float dtdx = dt / dx;
  const float rain_dt = s.rain_cont * dt;
  const float rain32_dt = s.rain32 * dt;
  const LiFaceConst fc = li_face_const(dt, dx);
  const bool has_comp = SRC == kLiSrcComp || (SRC == kLiSrcAny && p.h_comp != nullptr);
  const bool has_field = SRC == kLiSrcAny && p.rain_field != nullptr;
  const bool has_infil = SRC == kLiSrcAny && p.infil != nullptr;
  const int j = c0 + lane;  // this lane's column
  // row i0 - 2 of each array; rows outside the domain are never read or written
  const long long row0 = (long long)(i0 - 2) * nx, rowx = row0 + (i0 - 2);
  const float* __restrict__ h_in = p.hb[s.cur] + row0;
  const float* __restrict__ qx_in = p.qxb[s.cur] + rowx;
  const float* __restrict__ qy_in = p.qyb[s.cur] + row0;
  float* __restrict__ h_out = p.hb[s.cur ^ 1] + row0;
  float* __restrict__ qx_out = p.qxb[s.cur ^ 1] + rowx;
  float* __restrict__ qy_out = p.qyb[s.cur ^ 1] + row0;
  const float* __restrict__ z_in = p.z + row0;
  const float* __restrict__ n_in = p.n + row0;
  float* __restrict__ comp_io = has_comp ? p.h_comp + row0 : nullptr;
  const float* __restrict__ rain_in = has_field ? p.rain_field + row0 : nullptr;
  const float* __restrict__ infil_in = has_infil ? p.infil + row0 : nullptr;
  const float* __restrict__ d50_in = SED != 0 ? p.d50 + row0 : nullptr;
  float* __restrict__ six = SED != 0 ? p.qs_int_x + rowx : nullptr;
  float* __restrict__ scx = SED != 0 ? p.qs_comp_x + rowx : nullptr;
  float* __restrict__ siy = SED != 0 ? p.qs_int_y + row0 : nullptr;
  float* __restrict__ scy = SED != 0 ? p.qs_comp_y + row0 : nullptr;
  const bool in = !EDGE || (j >= 0 && j < nx);
  const bool face = !EDGE || (j >= 1 && j < nx);  // the x-face on this cell's west side is an inner face
  const bool own = in && lane >= kLiHalo && lane < 32 - kLiHalo;
  // x-face nx, the domain's east edge, goes with the last cell's strip
  const bool own_face = own || (EDGE && j == nx && lane > kLiHalo && lane <= 32 - kLiHalo);

  // carried rows: 1 is row r - 1 (faces unlimited), 2 is row r - 2 (faces limited)
  float h1 = 0.0f, z1 = 0.0f, n1 = 0.0f, x1 = 0.0f, y1 = 0.0f;
  float h2 = 0.0f, b2 = 1.0f, net2 = 0.0f, xl2 = 0.0f, xr2 = 0.0f, y2 = 0.0f;
  bool lim2 = false;  // whether any cell of row r - 2 has a beta below 1
  float fx1 = 0.0f, nx1 = 0.0f, fy1 = 0.0f, ny1 = 0.0f, g1 = 0.0f;  // bedload: face depths, roughness, grain size
  const float* lane_row = &ring.row[lane];
  const unsigned lane_dst = static_cast<unsigned>(__cvta_generic_to_shared(lane_row));
  // Start the copies of iteration r, into the row at `st` floats: row r of the state,
  // row r - 1 of the bedload operands and row r - 2 of the sources. A halo lane's
  // operands may be rewritten by their owner meanwhile; what it computes is not used.
  auto fetch = [&](int r, int id, int st) {
    const unsigned dst = lane_dst + st * 4;
    const int idx = id + (r - i0 + 2), id1 = id - nx, idx1 = idx - nx - 1, id2 = id1 - nx;
    const bool row = !EDGE || (r >= 0 && r < ny), row1 = !EDGE || (r - 1 >= 0 && r - 1 < ny);
    const bool row2 = !EDGE || (r - 2 >= i0 && r - 2 < i1);
    const float* z = p.z;
    copy_word<0, EDGE>(dst, h_in + id, row && in, z);
    copy_word<1, EDGE>(dst, z_in + id, row && in, z);
    copy_word<2, EDGE>(dst, n_in + id, row && in, z);
    copy_word<3, EDGE>(dst, qx_in + idx, row && face, z);
    copy_word<4, EDGE>(dst, qy_in + id, row && in && r >= 1, z);
    if (has_comp) copy_word<Ring::kComp, EDGE>(dst, comp_io + id2, row2 && in, z);
    if (has_field) copy_word<Ring::kRain, EDGE>(dst, rain_in + id2, row2 && in, z);
    if (has_infil) copy_word<Ring::kInfil, EDGE>(dst, infil_in + id2, row2 && in, z);
    if constexpr (SED != 0) {
      copy_word<Ring::kD50, EDGE>(dst, d50_in + id1, row1 && in, z);
      copy_word<Ring::kD50 + 1, EDGE>(dst, six + idx1, row1 && face, z);
      copy_word<Ring::kD50 + 2, EDGE>(dst, scx + idx1, row1 && face, z);
      copy_word<Ring::kD50 + 3, EDGE>(dst, siy + id1, row1 && in && r >= 2, z);
      copy_word<Ring::kD50 + 4, EDGE>(dst, scy + id1, row1 && in && r >= 2, z);
    }
    cp_async_commit();
  };
  int id = j;  // element (r, j) relative to row i0 - 2
  int st = 0;  // the staged row of iteration r, in floats
  fetch(i0 - 2, id, 0);
  // MAIN: every row this iteration completes is the chunk's own; the iterations at the
  // chunk's ends check.
  auto iterate = [&](int r, auto main_tag) {
    constexpr bool MAIN = decltype(main_tag)::value;
    const int id1 = id - nx, id2 = id1 - nx;
    // the row read in the previous iteration makes place for the next (one past the last
    // this chunk needs is refused by the bounds checks, or read and not used)
    if (!EDGE || r <= i1)
      fetch(r + 1, id + nx, st ^ Ring::kStage);
    else
      cp_async_commit();
    cp_async_wait<1>();
    const float* now = lane_row + st;
    const float h0 = now[0], z0 = now[32], n0 = now[64];
    float qo[2] = {now[96], now[128]};  // the x-face, then the y-face
    float g_comp = has_comp ? now[Ring::kComp * 32] : 0.0f;
    const float g_rain = has_field ? now[Ring::kRain * 32] : 0.0f;
    const float g_inf = has_infil ? now[Ring::kInfil * 32] : 0.0f;
    st ^= Ring::kStage;
    id += nx;
    const float e0 = h0 + z0;  // local_inertial.py:61-69
    const bool upd = MAIN || (r - 2 >= i0 && r - 2 < i1);
    const bool row1 = MAIN || (r - 1 >= i0 && r - 1 < i1);  // row r - 1's faces are this chunk's
    const int f1 = id1 + (r - 1 - i0 + 2);                  // x-face (r - 1, j)

    // unlimited faces (local_inertial.py:72-129); boundary faces stay 0, which is the
    // closed boundary (boundaries.py:223-241). The larger bed is a plain maximum: where
    // a bed is not a number, so is the surface on its side.
    const float ew = west_of(e0), zw = west_of(z0), nw = west_of(n0);
    const float e1 = h1 + z1;
    const float el[2] = {ew, e1}, er[2] = {e0, e0};
    const float hf[2] = {rmax(ew, e0) - fmaxf(zw, z0), rmax(e1, e0) - fmaxf(z1, z0)};
    const float nf[2] = {0.5f * (nw + n0), 0.5f * (n1 + n0)};
    const bool on[2] = {face && (!EDGE || (r >= 0 && r < ny)), in && (!EDGE || (r >= 1 && r < ny))};
    float q[2];
    li_faces<2>(qo, el, er, hf, nf, on, fc, q);

    // donor-cell beta of row r - 1 (local_inertial.py:197-239): the sum of its outgoing
    // discharges, and h / (dtdx sum) clamped to [0, 1] where it goes below 1. A quotient
    // of h >= out_depth is not below 1, so a warp none of whose cells could run dry, in
    // this row or the one above, leaves its faces as they are.
    const float xe = east_of(x1);
    const float out_depth = dtdx * (fmaxf(-x1, 0.0f) + fmaxf(xe, 0.0f) + fmaxf(-y1, 0.0f) + fmaxf(q[1], 0.0f));
    const bool lim1 = s.limit && __any_sync(kFullWarp, (out_depth > 0.0f) & !(h1 >= out_depth));
    float xl = x1, yl = y1;
    if (lim1 || lim2) {
      const bool out = lim1 && out_depth > 0.0f;
      const float ratio = div_if(out, h1, out_depth);
      const float b1 = out ? rclamp(ratio, 0.0f, 1.0f) : 1.0f;
      const float bw = west_of(b1);
      // scale each face by its donor's beta (:242-263): a zero face keeps its bits under
      // either (beta is in [0, 1]), so the domain's edge faces need no case
      xl = x1 * (x1 > 0.0f ? bw : b1);
      yl = y1 * (y1 > 0.0f ? b2 : b1);
      b2 = b1;
    }
    lim2 = lim1;
    const float xr = east_of(xl);
    if (row1 && own_face) qx_out[f1] = xl;
    if ((row1 || (EDGE && r - 1 == ny)) && own) qy_out[id1] = yl;  // and the domain's south edge
    if constexpr (SED != 0) {  // sediment.py:218-273 on the limited faces of row r - 1
      const float g0 = now[Ring::kD50 * 32], gw = west_of(g0);
      if (row1 && own && face) {
        float tot = now[(Ring::kD50 + 1) * 32], comp = now[(Ring::kD50 + 2) * 32];
        kahan_add(tot, comp, face_capacity(xl, fx1, fx1, nx1, 0.5f * (gw + g0)) * dt);
        six[f1] = tot;
        scx[f1] = comp;
      }
      if (row1 && own && (!EDGE || r - 1 >= 1)) {
        float tot = now[(Ring::kD50 + 3) * 32], comp = now[(Ring::kD50 + 4) * 32];
        kahan_add(tot, comp, face_capacity(yl, fy1, fy1, ny1, 0.5f * (g1 + g0)) * dt);
        siy[id1] = tot;
        scy[id1] = comp;
      }
      g1 = g0;
      fx1 = hf[0];
      nx1 = nf[0];
      fy1 = hf[1];
      ny1 = nf[1];
    }

    // continuity, areal sources, infiltration and open-edge sinks of row r - 2
    const bool ok = upd && own;
    const float net = net2 - yl;
    float h = h2 + dtdx * net + rain_dt;  // local_inertial.py:150-151
    if (has_comp) {
      if (!has_field)
        kahan_add(h, g_comp, rain32_dt);  // sources.py:85-101
      else
        kahan_add(h, g_comp, g_rain * s.scale32 * dt);  // sources.py:104-121
      if (ok) comp_io[id2] = g_comp;
    } else if (has_field) {
      h = h + g_rain * s.scale32 * dt;  // local_inertial.py:154-167
    }
    if (has_infil) {  // local_inertial.py:170-194
      const float avail = h;
      float inf = g_inf * dt;
      if (inf > avail) inf = avail;
      if (inf < 0.0f) inf = 0.0f;
      h = avail - inf;
      if (ok) loss += (double)avail - (double)h;
    }
    if (EDGE && ok) {  // boundaries.py:259-318, launched west, east, north, south
      const int gi = r - 2;
      const float avail0 = h;
      if (p.bc[RB_EDGE_WEST] == RB_BC_OPEN && nx > 1 && j == 0) h = drain(h, rmax(-xr2, 0.0f), s.dxdt);
      const float avail1 = h;
      if (p.bc[RB_EDGE_EAST] == RB_BC_OPEN && nx > 1 && j == nx - 1) h = drain(h, rmax(xl2, 0.0f), s.dxdt);
      const float avail2 = h;
      if (p.bc[RB_EDGE_NORTH] == RB_BC_OPEN && ny > 1 && gi == 0) h = drain(h, rmax(-yl, 0.0f), s.dxdt);
      const float avail3 = h;
      if (p.bc[RB_EDGE_SOUTH] == RB_BC_OPEN && ny > 1 && gi == ny - 1) h = drain(h, rmax(y2, 0.0f), s.dxdt);
      loss += ((double)avail0 - (double)avail1) + ((double)avail1 - (double)avail2) +
              ((double)avail2 - (double)avail3) + ((double)avail3 - (double)h);
    }
    if (ok) h_out[id2] = h;
    // an inner strip's halo lanes are left out after the loop
    const bool count = (MAIN && !EDGE) || ok;
    hmax = fmaxf(hmax, count ? h : 0.0f);
    bad |= count & !(fabsf(h) <= FLT_MAX);
    net2 = xl - xr + yl;
    if constexpr (EDGE) {
      xl2 = xl;
      xr2 = xr;
      y2 = yl;
    }
    h2 = h1;
    h1 = h0;
    z1 = z0;
    n1 = n0;
    x1 = q[0];
    y1 = q[1];
  };
  if constexpr (EDGE) {
#pragma unroll 1
    for (int r = i0 - 2; r <= i1 + 1; r++) iterate(r, std::false_type{});
  } else {
    int r = i0 - 2;
#pragma unroll 1
    for (; r < i0 + 2; r++) iterate(r, std::false_type{});
#if defined(RB_FAST_MATH)
#pragma unroll 2  // without the moves of the carried rows; the exact body is too long for it
#else
#pragma unroll 1
#endif
    for (; r <= i1; r++) iterate(r, std::true_type{});
    iterate(r, std::false_type{});
    // the copy ahead of the last row: nothing may land in the next block's shared memory.
    // (Not starting it instead: the 8192^2 reach 0.5 % slower.)
    cp_async_wait<0>();
    if (!own) hmax = 0.0f, bad = false;
  }
}

// One block's strip and chunk. `order` counts chunks as they are started: the last one
// runs second, since the domain's top and bottom chunks are the slow ones.
template <int SED, int SRC>
__device__ __forceinline__ void li_stream_block(const LiParams& p, int strip, int order, int chunks, size_t slot,
                                                int rows, LiRing<SED, SRC>& ring) {
  LiStepScalars s;
  if (!li_scalars(p, s)) return;
  const int c0 = strip * kLiStreamCols - kLiHalo;
  const int chunk = order == 1 ? chunks - 1 : (order > 1 ? order - 1 : 0);
  const int i0 = chunk * rows, i1 = min(p.ny, i0 + rows);
  double loss = 0.0;
  float hmax = 0.0f;
  bool bad = false;
  // inner strips read rows i0 - 4 (sources of the rows above) .. i1 + 2 (the copy ahead)
  if (c0 >= 1 && c0 + 32 <= p.nx && i0 >= 4 && i1 + 3 <= p.ny)
    li_stream_strip<SED, SRC, false>(p, s, c0, i0, i1, ring, loss, hmax, bad);
  else
    li_stream_strip<SED, SRC, true>(p, s, c0, i0, i1, ring, loss, hmax, bad);
  pdl_trigger();
  const int lane = threadIdx.x;
  if (p.ledger != nullptr) {
    const double t = warp_sum(loss);
    if (lane == 0) ledger_add(p.ledger + 2 * slot, t);
  }
  if (p.hmax_key != nullptr) {
    hmax = warp_max(hmax);
    if (lane == 0) atomicMax(p.hmax_key, max_key(hmax));
  }
  if (bad) flag_error(p.err, RB_DEVERR_NONFINITE);
}

// One warp a block: a block's warps would wait for its slowest strip before the
// reductions above (14 % of the warp cycles with four warps a block).
template <int SED, int SRC>
__global__ void __launch_bounds__(32, kLiStreamWarps) li_stream_kernel(const LiParams p, int rows) {
  __shared__ LiRing<SED, SRC> ring;
  pdl_wait();
  li_stream_block<SED, SRC>(p, blockIdx.x, blockIdx.y, gridDim.y, (size_t)blockIdx.y * gridDim.x + blockIdx.x, rows,
                            ring);
}

// Rows a warp walks: as many warps as the GPU holds at once, within 8 .. 48 (four rows
// above and below a chunk are overhead, and longer chunks leave the last wave uneven:
// 2048^2 fast 57.2 / 56.0 / 73.6 us for 22 / 43 / 86 rows, 4096^2 172.7 / 170.3 / 175.3).
static int li_stream_rows(int ny, int nx) {
  constexpr long long kWarps = 148LL * kLiStreamWarps;
  const long long strips = (nx + kLiStreamCols - 1) / kLiStreamCols;
  const long long rows = (ny * strips + kWarps - 1) / kWarps;
  return (int)(rows < 8 ? 8 : (rows > 48 ? 48 : rows));
}

// Whether the streaming kernel takes this domain. A warp walks its rows one after another,
// and a small domain has too few warps to hide that (us per step, tiles / streaming --
// exact: 1024^2 32.7 / 32.9, 1200^2 42.2 / 39.5, 1531 x 1017 with rain field and
// infiltration 47.5 / 48.1, 1380^2 53.1 / 48.6, 2048^2 118 / 92; fast: 512^2 18.0 / 18.2,
// 1024^2 28.9 / 22.9, 1531 x 1017 39.4 / 33.2, 2048^2 89.6 / 54.3, 4096^2 322 / 170). One
// limit serves all sources and lies above the largest domain on which the tiles won, that
// with rain field and infiltration (1.56 M cells); a plain 1200^2 would gain 6 % by
// streaming. The ledger has a slot per 32 x 8 cells, enough for one per strip and chunk
// except on narrow or flat domains.
#if defined(RB_FAST_MATH)
constexpr long long kLiStreamCells = 400000;
#else
constexpr long long kLiStreamCells = 1700000;
#endif
static bool li_stream_takes(const LiParams& p) {
  if (p.cw != nullptr || (long long)p.ny * p.nx < kLiStreamCells) return false;
  const int rows = li_stream_rows(p.ny, p.nx);
  const long long blocks = (long long)((p.nx + kLiStreamCols - 1) / kLiStreamCols) * ((p.ny + rows - 1) / rows);
  if (blocks > (long long)((p.nx + 31) / 32) * ((p.ny + 7) / 8)) return false;
  return (p.ny + rows - 1) / rows <= 65535 && (long long)(rows + 8) * (p.nx + 1) < (1LL << 31);
}

static cudaError_t launch_li_stream(const LiParams& p, cudaStream_t s) {
  const int rows = li_stream_rows(p.ny, p.nx);
  const dim3 grid((p.nx + kLiStreamCols - 1) / kLiStreamCols, (p.ny + rows - 1) / rows), block(32);
  if (p.d50 != nullptr) return launch_chain(li_stream_kernel<1, kLiSrcAny>, grid, block, 0, s, p, rows);
  if (p.rain_field != nullptr || p.infil != nullptr)
    return launch_chain(li_stream_kernel<0, kLiSrcAny>, grid, block, 0, s, p, rows);
  if (p.h_comp != nullptr) return launch_chain(li_stream_kernel<0, kLiSrcComp>, grid, block, 0, s, p, rows);
  return launch_chain(li_stream_kernel<0, kLiSrcNone>, grid, block, 0, s, p, rows);
}

#if !defined(RB_FAST_MATH)
// The larger domains of an ensemble in one launch: together they fill the GPU where each
// alone would leave part of its last wave, or all of it, idle (a mix of 20 domains of 128^2
// to 1364^2, us per step: 545 with a launch for each of the three largest and a work-list of
// tiles for the rest, 460 with a launch per scheme and stage).
template <int SRC>
__global__ void __launch_bounds__(32, kLiStreamWarps)
    ens_li_stream_kernel(const __grid_constant__ StreamGroup<LiParams> g) {
  __shared__ LiRing<0, SRC> ring;
  pdl_wait();
  int d = 0;
  while ((int)blockIdx.x >= g.first[d + 1]) d++;
  const LiParams& p = g.p[d];
  const int strips = (p.nx + kLiStreamCols - 1) / kLiStreamCols;
  const int b = blockIdx.x - g.first[d];
  li_stream_block<0, SRC>(p, b % strips, b / strips, (p.ny + g.rows - 1) / g.rows, (size_t)b, g.rows, ring);
}

constexpr int kEnsLiMinRows = 12;  // 28 x 12 cells a block: what the ledger's slots allow
bool ens_li_stream_fits(const LiParams& p) {
  const long long blocks = (long long)((p.nx + kLiStreamCols - 1) / kLiStreamCols) *
                           ((p.ny + kEnsLiMinRows - 1) / kEnsLiMinRows);
  return p.d50 == nullptr && p.cw == nullptr && blocks <= (long long)((p.nx + 31) / 32) * ((p.ny + 7) / 8) &&
         (48 + 8LL) * (p.nx + 1) < (1LL << 31) && blocks < (1LL << 31) / kStreamGroup;
}

cudaError_t ens_li_stream_launch(const LiParams* p, int n, cudaStream_t s) {
  const int groups = (n + kStreamGroup - 1) / kStreamGroup;
  for (int k = 0; k < groups; k++) {
    const int d0 = (int)((long long)n * k / groups), m = (int)((long long)n * (k + 1) / groups) - d0;
    StreamGroup<LiParams> g{};
    long long strip_rows = 0;
    bool any = false, comp = true;
    for (int d = 0; d < m; d++) {
      const LiParams& q = g.p[d] = p[d0 + d];
      strip_rows += (long long)((q.nx + kLiStreamCols - 1) / kLiStreamCols) * q.ny;
      any |= q.rain_field != nullptr || q.infil != nullptr || (q.h_comp != nullptr) != (g.p[0].h_comp != nullptr);
      comp = comp && q.h_comp != nullptr;
    }
    const long long rows = (strip_rows + 148LL * kLiStreamWarps - 1) / (148LL * kLiStreamWarps);
    g.rows = (int)(rows < kEnsLiMinRows ? kEnsLiMinRows : (rows > 48 ? 48 : rows));
    for (int d = 0; d < kStreamGroup; d++)
      g.first[d + 1] = g.first[d] + (d < m ? ((g.p[d].nx + kLiStreamCols - 1) / kLiStreamCols) *
                                                 ((g.p[d].ny + g.rows - 1) / g.rows)
                                           : 0);
    const dim3 grid(g.first[m]), block(32);
    const cudaError_t e = any    ? launch_chain(ens_li_stream_kernel<kLiSrcAny>, grid, block, 0, s, g)
                          : comp ? launch_chain(ens_li_stream_kernel<kLiSrcComp>, grid, block, 0, s, g)
                                 : launch_chain(ens_li_stream_kernel<kLiSrcNone>, grid, block, 0, s, g);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
#endif
