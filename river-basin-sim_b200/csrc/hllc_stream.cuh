// hllc_stream.cuh -- one Heun stage of the HLLC step as a row-streaming kernel.
//
// Included by hllc_step.cu inside its arithmetic namespace, after the face functions.
//
// A warp owns a strip of 32 columns (a cell a lane) and walks down the rows of its chunk.
// Rows above live in registers and the cells to the left and right come by warp shuffle,
// so each cell is reconstructed once per direction and each face solved once per strip,
// with no shared memory traffic between threads and no barrier. Row r enters at
// iteration r:
//   r    : primitives and their differences to row r - 1
//   r - 1: reconstruction along y; the y-face above it (with the southern values kept
//          from row r - 2); reconstruction along x and its x-faces
//   r - 2: its four faces are known now: the momentum divergence, the bed source, beta;
//          its x-faces and the y-face above it are limited
//   r - 3: its four limited mass faces are known now: the Heun update, stored
// The outer three columns on either side of a strip and three rows above and below a
// chunk are computed by the neighbouring warps as well and stored by them.
#pragma once

constexpr int kHllcHalo = 3;
constexpr int kHllcStreamCols = 32 - 2 * kHllcHalo;  // columns a strip stores

// A warp's staging area: the row in use and the one on its way, each lane's word of
// every array its iteration reads. Arrays: h, hu, hv, z of row r; of row r - 3 the
// stage's momenta, then (stage 2) U^n and the roughness, then the sources.
template <int STAGE, int SRC>
struct HllcRing {
  static constexpr int kMom = 4, kOld = 6, kSrc = 10;
  static constexpr int kStage = (STAGE == 1 ? 8 : 16) * 32;  // floats a row, a power of two
  alignas(16) float row[2 * kStage];
};

// One cell's values along a direction: surface, bed, normal and transverse velocity.
struct Quad {
  float e, z, n, t;
};
__device__ __forceinline__ Quad operator-(const Quad& a, const Quad& b) {
  return Quad{a.e - b.e, a.z - b.z, a.n - b.n, a.t - b.t};
}
__device__ __forceinline__ Quad west_of(const Quad& q) {
  return Quad{west_of(q.e), west_of(q.z), west_of(q.n), west_of(q.t)};
}
__device__ __forceinline__ Quad east_of(const Quad& q) {
  return Quad{east_of(q.e), east_of(q.z), east_of(q.n), east_of(q.t)};
}

// any_face_flux's operands for the face: what goes into the Riemann solve (the ghost
// states of an edge face included) and the depths of the bed-slope corrections.
struct FaceOperands {
  float hl, ul, vl, hr, ur, vr;
  float h_l, h_r, hl_star, hr_star;
};
__device__ __forceinline__ FaceOperands face_operands(const Quad& L, const Quad& R, int kind, bool low, const Cell& e,
                                                      float stage) {
  FaceOperands f;
  const float z_star = rmax(L.z, R.z);
  f.h_l = fmaxf(L.e - L.z, 0.0f);
  f.h_r = fmaxf(R.e - R.z, 0.0f);
  f.hl = f.hl_star = fmaxf(L.e - z_star, 0.0f);
  f.hr = f.hr_star = fmaxf(R.e - z_star, 0.0f);
  f.ul = L.n;
  f.vl = L.t;
  f.ur = R.n;
  f.vr = R.t;
  if (kind != RB_BC_OPEN) {
    const bool closed = kind == RB_BC_CLOSED;
    const float h_g = rmax(stage - e.z, 0.0f);
    f.hl = (!closed && low) ? h_g : e.h;
    f.hr = (!closed && !low) ? h_g : e.h;
    f.ul = (closed && low) ? -e.un : e.un;
    f.ur = (closed && !low) ? -e.un : e.un;
    f.vl = e.ut;
    f.vr = e.ut;
  }
  return f;
}
struct FaceFlux {
  float h, l, r, t;  // mass, normal momentum to the left and to the right cell, transverse
};
__device__ __forceinline__ FaceFlux face_flux(const FaceOperands& f, float f0, float f1, float f2, int kind, bool low) {
  if (kind != RB_BC_OPEN) return FaceFlux{f0, low ? 0.0f : f1, low ? f1 : 0.0f, f2};
  const float g = kG;
  return FaceFlux{f0, f1 + 0.5f * g * (f.h_l * f.h_l - f.hl_star * f.hl_star),
                  f1 + 0.5f * g * (f.h_r * f.h_r - f.hr_star * f.hr_star), f2};
}

// recon() from the differences to the lower (dm) and upper (dp) neighbour: the same
// operations on the same operands.
__device__ __forceinline__ Rec recon_diff(const Quad& c, const Quad& dm, const Quad& dp, bool any_dry) {
  const float dry = any_dry ? 0.0f : 1.0f;
  const float hw = 0.5f * dry;
  const float me = minmod(dm.e, dp.e), mz = minmod(dm.z, dp.z);
  const float mn = minmod(dm.n, dp.n), mt = minmod(dm.t, dp.t);
  Rec r;
  r.eE = c.e + hw * me;
  r.eW = c.e - hw * me;
  r.zE = c.z + hw * mz;
  r.zW = c.z - hw * mz;
  r.nE = c.n + hw * mn;
  r.nW = c.n - hw * mn;
  r.tE = c.t + hw * mt;
  r.tW = c.t - hw * mt;
  r.sz = dry * mz;
  return r;
}

// Rows [i0, i1) of the strip whose first column (lane 0) is c0. EDGE: the strip or its
// halo may reach a domain edge (clamped indices, edge faces, banking); the other
// instantiation is for strips whose every staged cell lies inside. Element offsets are
// 32-bit, relative to the row six above the chunk (the launcher keeps a chunk below 2^31).
template <int STAGE, int SRC, bool EDGE>
__device__ __forceinline__ void hllc_stream_strip(const HllcParams& p, const HllcStageScalars& s, int c0, int i0,
                                                  int i1, HllcRing<STAGE, SRC>& ring, double& loss, float& smax,
                                                  bool& bad) {
  using Ring = HllcRing<STAGE, SRC>;
  const int lane = threadIdx.x & 31;
  const int ny = p.ny, nx = p.nx;
  const float dt = s.dt, dx = p.dx32;
  const float dtdx = dt / dx, inv_dx = 1.0f / dx;
  const float g = kG;
  const int j = c0 + lane;  // this lane's column
  const long long row0 = EDGE ? 0 : (long long)(i0 - 6) * nx;
  const float* __restrict__ h_s = (STAGE == 1 ? p.hb[s.cur] : p.h1) + row0;
  const float* __restrict__ hu_s = (STAGE == 1 ? p.hub[s.cur] : p.hu1) + row0;
  const float* __restrict__ hv_s = (STAGE == 1 ? p.hvb[s.cur] : p.hv1) + row0;
  const float* __restrict__ z_in = p.z + row0;
  const float* __restrict__ h_n = p.hb[s.cur] + row0;
  const float* __restrict__ hu_n = p.hub[s.cur] + row0;
  const float* __restrict__ hv_n = p.hvb[s.cur] + row0;
  const float* __restrict__ n_in = p.n + row0;
  float* __restrict__ h_out = (STAGE == 1 ? p.h1 : p.hb[s.cur ^ 1]) + row0;
  float* __restrict__ hu_out = (STAGE == 1 ? p.hu1 : p.hub[s.cur ^ 1]) + row0;
  float* __restrict__ hv_out = (STAGE == 1 ? p.hv1 : p.hvb[s.cur ^ 1]) + row0;
  const bool has_comp = SRC != 0 && p.h_comp != nullptr;
  const bool has_field = SRC != 0 && p.rain_field != nullptr;
  const bool has_infil = SRC != 0 && p.infil != nullptr;
  const bool in = !EDGE || (j >= 0 && j < nx);
  const bool own = in && lane >= kHllcHalo && lane < 32 - kHllcHalo;
  const int kind_x = !EDGE ? RB_BC_OPEN : (j == 0 ? p.bc[RB_EDGE_WEST] : (j == nx ? p.bc[RB_EDGE_EAST] : RB_BC_OPEN));
  const float stage_x = j == 0 ? s.stage[RB_EDGE_WEST] : s.stage[RB_EDGE_EAST];

  const unsigned near_lanes = lane == 0 ? 3u : 7u << (lane - 1);  // this lane and its neighbours
  const float* lane_row = &ring.row[lane];
  const unsigned lane_dst = static_cast<unsigned>(__cvta_generic_to_shared(lane_row));
  const int jc = EDGE ? min(max(j, 0), nx - 1) : j;
  // Start the copies of iteration r into the row at `st` floats: row r of the state and
  // row r - 3 of the update's operands. Indices outside the domain are clamped to it
  // (the reference's _cget transmissive ghosts). A halo lane's h_comp may be rewritten by
  // its owner meanwhile; what it computes is not used.
  auto fetch = [&](int r, int st) {
    const unsigned dst = lane_dst + st * 4;
    const long long id = EDGE ? (long long)min(max(r, 0), ny - 1) * nx + jc : (long long)((r - i0 + 6) * nx + jc);
    const long long id3 = EDGE ? (long long)min(max(r - 3, 0), ny - 1) * nx + jc : (long long)((r - i0 + 3) * nx + jc);
    copy_word<0, false>(dst, h_s + id, true, nullptr);
    copy_word<1, false>(dst, hu_s + id, true, nullptr);
    copy_word<2, false>(dst, hv_s + id, true, nullptr);
    copy_word<3, false>(dst, z_in + id, true, nullptr);
    copy_word<Ring::kMom, false>(dst, hu_s + id3, true, nullptr);
    copy_word<Ring::kMom + 1, false>(dst, hv_s + id3, true, nullptr);
    if constexpr (STAGE == 2) {
      copy_word<Ring::kOld, false>(dst, h_n + id3, true, nullptr);
      copy_word<Ring::kOld + 1, false>(dst, hu_n + id3, true, nullptr);
      copy_word<Ring::kOld + 2, false>(dst, hv_n + id3, true, nullptr);
      copy_word<Ring::kOld + 3, false>(dst, n_in + id3, true, nullptr);
      if (has_comp) copy_word<Ring::kSrc, false>(dst, p.h_comp + row0 + id3, true, nullptr);
      if (has_field) copy_word<Ring::kSrc + 1, false>(dst, p.rain_field + row0 + id3, true, nullptr);
      if (has_infil) copy_word<Ring::kSrc + 2, false>(dst, p.infil + row0 + id3, true, nullptr);
    }
    cp_async_commit();
  };

  // carried rows: 1 is row r - 1, 2 is row r - 2, 3 is row r - 3
  float h1 = 1.0f, h2 = 1.0f, h3 = 1.0f;
  Quad c1{0, 0, 0, 0}, d1{0, 0, 0, 0};      // row r - 1 in the y frame, and its difference to row r - 2
  bool dry1 = false, dry2 = false;
  Quad s2{0, 0, 0, 0};                      // southern values of row r - 2
  Quad c2{0, 0, 0, 0};                      // row r - 2 (edge faces only)
  float fw2 = 0, fe2 = 0, a2 = 0, b2 = 0, sx2 = 0;  // row r - 2: x mass faces, x momentum differences, x bed source
  float fn2 = 0, frn2 = 0, ftn2 = 0, hm2 = 0, sz2 = 0;  // its northern face, northern depth, bed slope
  float qw3 = 0, qe3 = 0, qn3 = 0, be3 = 1.0f, dhu3 = 0, dhv3 = 0;  // row r - 3: limited faces, beta, rates
  bool lim3 = false;
  int st = 0;
  fetch(i0 - 3, 0);
  auto iterate = [&](int r, auto main_tag) {
    constexpr bool MAIN = decltype(main_tag)::value;
    if (!EDGE || r < i1 + 2)
      fetch(r + 1, st ^ Ring::kStage);
    else
      cp_async_commit();
    cp_async_wait<1>();
    const float* now = lane_row + st;
    st ^= Ring::kStage;
    const float h0 = now[0], z0 = now[96];
    float u0, v0;
    bool odd0 = false;
    primitives_near(h0, now[32], now[64], u0, v0, odd0);
#if !defined(RB_FAST_MATH)
    if (__any_sync(kFullWarp, odd0)) primitives_any(h0, now[32], now[64], u0, v0);
#endif
    const Quad c0q{h0 + z0, z0, v0, u0};  // the y frame: normal v, transverse u
    const Quad d0 = c0q - c1;
    const bool dry0 = h0 <= kHDry;

    // row r - 1 along y, and the y-face between rows r - 2 and r - 1 (face row r - 1)
    const Rec ry = recon_diff(c1, d1, d0, dry0 || dry1 || dry2);
    FaceFlux fy{0, 0, 0, 0}, fx{0, 0, 0, 0};
    float hl = 0, hr = 0, kr = 0, sxx = 0, hpx = 0;
    if (MAIN || r >= i0) {
      const int fi = r - 1;
      const int kind_y =
          !EDGE ? RB_BC_OPEN : (fi == 0 ? p.bc[RB_EDGE_NORTH] : (fi == ny ? p.bc[RB_EDGE_SOUTH] : RB_BC_OPEN));
      const Cell ey = fi == 0 ? Cell{h1, c1.n, c1.t, c1.z} : Cell{h2, c2.n, c2.t, c2.z};
      const FaceOperands oy = face_operands(s2, Quad{ry.eW, ry.zW, ry.nW, ry.tW}, kind_y, fi == 0, ey,
                                            fi == 0 ? s.stage[RB_EDGE_NORTH] : s.stage[RB_EDGE_SOUTH]);
      // row r - 1 along x, and the x-face on this cell's west side
      const Quad x1{c1.e, c1.z, c1.t, c1.n};
      const Quad dw = x1 - west_of(x1), de = east_of(dw);
      const unsigned dry_mask = __ballot_sync(kFullWarp, dry1);
      const Rec rx = recon_diff(x1, dw, de, (dry_mask & near_lanes) != 0);
      const Quad wE = west_of(Quad{rx.eE, rx.zE, rx.nE, rx.tE});
      Cell ex{h1, x1.n, x1.t, x1.z};
      if constexpr (EDGE) {
        if (c0 + 32 > nx) {  // the east edge's cell is the one to the west of its face
          const Cell w{west_of(h1), west_of(x1.n), west_of(x1.t), west_of(x1.z)};
          if (j == nx) ex = w;
        }
      }
      const FaceOperands ox =
          face_operands(wE, Quad{rx.eW, rx.zW, rx.nW, rx.tW}, kind_x, j == 0, ex, stage_x);
      float y0, y1, y2, x0, x1f, x2;
      bool odd = false;
      F2 p0, p1, p2;
      hllc_near2(F2{oy.hl, ox.hl}, F2{oy.ul, ox.ul}, F2{oy.vl, ox.vl}, F2{oy.hr, ox.hr}, F2{oy.ur, ox.ur},
                 F2{oy.vr, ox.vr}, p0, p1, p2, odd);
      y0 = p0.x, y1 = p1.x, y2 = p2.x, x0 = p0.y, x1f = p1.y, x2 = p2.y;
#if !defined(RB_FAST_MATH)
      if (__any_sync(kFullWarp, odd)) {
        hllc_flux_any(oy.hl, oy.ul, oy.vl, oy.hr, oy.ur, oy.vr, y0, y1, y2);
        hllc_flux_any(ox.hl, ox.ul, ox.vl, ox.hr, ox.ur, ox.vr, x0, x1f, x2);
      }
#endif
      fy = face_flux(oy, y0, y1, y2, kind_y, fi == 0);
      fx = face_flux(ox, x0, x1f, x2, kind_x, j == 0);
      hl = oy.h_l;
      hr = oy.h_r;
      kr = ox.h_r;
      hpx = fmaxf(rx.eE - rx.zE, 0.0f);
      sxx = rx.sz;
    }

    // row r - 2: rates of the momenta (hllc.py:776-847), beta (:700-736), limited faces
    const float srcy = -g * 0.5f * (hl + hm2) * sz2;
    const float dhu2 = (-(a2 + (fy.t - ftn2)) + sx2) * inv_dx;
    const float dhv2 = (-((fy.l - frn2) + b2) + srcy) * inv_dx;
    const float out_depth = dtdx * (fmaxf(-fw2, 0.0f) + fmaxf(fe2, 0.0f) + fmaxf(-fn2, 0.0f) + fmaxf(fy.h, 0.0f));
    const bool cell2 = !EDGE || (in && r - 2 >= 0 && r - 2 < ny);
    const bool lim2 = __any_sync(kFullWarp, cell2 & (out_depth > 0.0f) & !(h2 >= out_depth));
    float qw = fw2, qn = fn2, be2 = 1.0f;
    if (lim2 || lim3) {
      const bool out = lim2 && cell2 && out_depth > 0.0f;
      const float ratio = div_if(out, h2, out_depth);
      be2 = out ? rclamp(ratio, 0.0f, 1.0f) : 1.0f;
      const float bw = west_of(be2);
      qw = fw2 * (fw2 > 0.0f ? bw : be2);
      qn = fn2 * (fn2 > 0.0f ? be3 : be2);
    }
    const float qe = east_of(qw);

    // row r - 3: the Heun update
    if (MAIN) {
      const int gi = r - 3;
      const long long id3 = EDGE ? (long long)gi * nx + j : (long long)((r - i0 + 3) * nx + j);
      if (EDGE && own && p.ledger != nullptr) {  // hllc.py:638-677
        if (j == 0 && p.bc[RB_EDGE_WEST] != RB_BC_CLOSED) loss -= s.wt * (double)qw3;
        if (j == nx - 1 && p.bc[RB_EDGE_EAST] != RB_BC_CLOSED) loss += s.wt * (double)qe3;
        if (gi == 0 && p.bc[RB_EDGE_NORTH] != RB_BC_CLOSED) loss -= s.wt * (double)qn3;
        if (gi == ny - 1 && p.bc[RB_EDGE_SOUTH] != RB_BC_CLOSED) loss += s.wt * (double)qn;
      }
      const float dh = -((qe3 - qw3) + (qn - qn3)) * inv_dx;
      const float hus = now[Ring::kMom * 32], hvs = now[(Ring::kMom + 1) * 32];
      if constexpr (STAGE == 1) {  // hllc.py:850-878
        const float hh = fmaxf(h3 + dt * dh, 0.0f);
        const bool wet = hh > kHDry;
        const float hu1 = wet ? hus + dt * dhu3 : 0.0f;
        const float hv1 = wet ? hvs + dt * dhv3 : 0.0f;
        if (own) {
          h_out[id3] = hh;
          hu_out[id3] = hu1;
          hv_out[id3] = hv1;
        }
      } else {  // hllc.py:881-909, then friction :912-939, then sources :1350-1373
        float hh = fmaxf(0.5f * (now[Ring::kOld * 32] + h3 + dt * dh), 0.0f);
        const bool wet = hh > kHDry;
        float hu = wet ? 0.5f * (now[(Ring::kOld + 1) * 32] + hus + dt * dhu3) : 0.0f;
        float hv = wet ? 0.5f * (now[(Ring::kOld + 2) * 32] + hvs + dt * dhv3) : 0.0f;
        hllc_friction<true>(hh, wet, g * dt, now[(Ring::kOld + 3) * 32], hu, hv);
        if (SRC != 0 && s.rain_mode == 1) {
          float comp = now[Ring::kSrc * 32];
          kahan_add(hh, comp, s.rain32 * dt);
          if (own) p.h_comp[row0 + id3] = comp;
        } else if (s.rain_mode == 2) {
          hh = hh + s.rain32 * dt;  // hllc.py:942-945
        }
        if (has_field) {
          const float add = now[(Ring::kSrc + 1) * 32] * s.scale32 * dt;
          if (has_comp) {
            float comp = now[Ring::kSrc * 32];
            kahan_add(hh, comp, add);
            if (own) p.h_comp[row0 + id3] = comp;
          } else {
            hh = hh + add;
          }
        }
        if (has_infil) {  // local_inertial.py:170-194
          const float avail = hh;
          float inf = now[(Ring::kSrc + 2) * 32] * dt;
          if (inf > avail) inf = avail;
          if (inf < 0.0f) inf = 0.0f;
          hh = avail - inf;
          if (own) loss += (double)avail - (double)hh;
        }
        if (own) {
          h_out[id3] = hh;
          hu_out[id3] = hu;
          hv_out[id3] = hv;
        }
        const float sp = wave_speed<true>(hh, hu, hv);  // hllc.py:948-966 on the new state
        smax = fmaxf(smax, EDGE && !own ? 0.0f : sp);
        bad |= (!EDGE | own) & (!(fabsf(hh) <= FLT_MAX) | !(fabsf(hu) <= FLT_MAX) | !(fabsf(hv) <= FLT_MAX));
      }
    }
    qw3 = qw;
    qe3 = qe;
    qn3 = qn;
    be3 = be2;
    lim3 = lim2;
    dhu3 = dhu2;
    dhv3 = dhv2;
    fw2 = fx.h;
    fe2 = east_of(fx.h);
    a2 = east_of(fx.l) - fx.r;
    b2 = east_of(fx.t) - fx.t;
    sx2 = -g * 0.5f * (hpx + kr) * sxx;
    fn2 = fy.h;
    frn2 = fy.r;
    ftn2 = fy.t;
    hm2 = hr;
    sz2 = ry.sz;
    s2 = Quad{ry.eE, ry.zE, ry.nE, ry.tE};
    if constexpr (EDGE) c2 = c1;
    h3 = h2;
    h2 = h1;
    h1 = h0;
    dry2 = dry1;
    dry1 = dry0;
    d1 = d0;
    c1 = c0q;
  };
  int r = i0 - 3;
#pragma unroll 1
  for (; r < i0 + 3; r++) iterate(r, std::false_type{});
#if defined(RB_FAST_MATH)
#pragma unroll 2  // without half of the moves of the carried rows; the exact body is too long for it
#else
#pragma unroll 1
#endif
  for (; r <= i1 + 2; r++) iterate(r, std::true_type{});
  // the copy ahead of the last row: nothing may land in the next block's shared memory.
  // (Not starting it instead: 2048^2 lake 1.1 % slower, fast dam break 1.5 % faster.)
  cp_async_wait<0>();
  if (!EDGE && !own) smax = 0.0f, bad = false;
}

// One block's strip and chunk. `order` counts chunks as they are started: the last one
// runs second, since the domain's top and bottom chunks are the slow ones.
template <int STAGE, int SRC>
__device__ __forceinline__ void hllc_stream_block(const HllcParams& p, int strip, int order, int chunks, size_t slot,
                                                  int rows, HllcRing<STAGE, SRC>& ring) {
  HllcStageScalars s;
  if (!hllc_scalars(p, s)) return;
  const int c0 = strip * kHllcStreamCols - kHllcHalo;
  const int chunk = order == 1 ? chunks - 1 : (order > 1 ? order - 1 : 0);
  const int i0 = chunk * rows, i1 = min(p.ny, i0 + rows);
  double loss = 0.0;
  float smax = 0.0f;
  bool bad = false;
  // inner strips read rows i0 - 6 (operands of the rows above) .. i1 + 3 (the copy ahead)
  if (c0 >= 0 && c0 + 32 <= p.nx && i0 >= 6 && i1 + 4 <= p.ny)
    hllc_stream_strip<STAGE, SRC, false>(p, s, c0, i0, i1, ring, loss, smax, bad);
  else
    hllc_stream_strip<STAGE, SRC, true>(p, s, c0, i0, i1, ring, loss, smax, bad);
  pdl_trigger();
  const int lane = threadIdx.x;
  if (p.ledger != nullptr) {
    const double t = warp_sum(loss);
    if (lane == 0) ledger_add(p.ledger + 2 * slot, t);
  }
  if (STAGE == 2) {
    if (p.smax_key != nullptr) {
      smax = warp_max(smax);
      if (lane == 0) atomicMax(p.smax_key, max_key(smax));
    }
    if (bad) flag_error(p.err, RB_DEVERR_NONFINITE);
  }
}

// One warp a block (no sibling to wait for at the end), 16 resident per SM: at 20 and 24
// (96 and 80 registers) the schedulers have no more to issue and the spills show (2048^2
// dam break, faces one by one, us per step, fast / exact: 189.7 / 270 for 16, 198.8 / 296 for 20, 209.9 / 308
// for 24).
constexpr int kHllcStreamWarps = 16;
template <int STAGE, int SRC>
__global__ void __launch_bounds__(32, kHllcStreamWarps) hllc_stream_kernel(const HllcParams p, int rows) {
  __shared__ HllcRing<STAGE, SRC> ring;
  pdl_wait();
  hllc_stream_block<STAGE, SRC>(p, blockIdx.x, blockIdx.y, gridDim.y, (size_t)blockIdx.y * gridDim.x + blockIdx.x,
                                rows, ring);
}

// Rows a warp walks: two waves of the warps the GPU holds, within 11 .. 48: three rows
// above and below a chunk are overhead, and with one long wave the domain's edge strips,
// which check bounds, end last (2048^2 dam break, fast, us per step: 196 / 190 / 191 / 228
// for 19 / 28 / 35 / 48 rows).
static int hllc_stream_rows(int ny, int nx) {
  constexpr long long kWarps = 2LL * 148 * kHllcStreamWarps;
  const long long strips = (nx + kHllcStreamCols - 1) / kHllcStreamCols;
  const long long rows = (ny * strips + kWarps - 1) / kWarps;
  return (int)(rows < 11 ? 11 : (rows > 48 ? 48 : rows));
}

static cudaError_t launch_hllc_stream(const HllcParams& p, int stage, cudaStream_t s) {
  const int rows = hllc_stream_rows(p.ny, p.nx);
  const dim3 grid((p.nx + kHllcStreamCols - 1) / kHllcStreamCols, (p.ny + rows - 1) / rows), block(32);
  if (stage == 1) return launch_chain(hllc_stream_kernel<1, 0>, grid, block, 0, s, p, rows);
  const bool src = p.h_comp != nullptr || p.rain_field != nullptr || p.infil != nullptr;
  return src ? launch_chain(hllc_stream_kernel<2, 1>, grid, block, 0, s, p, rows)
             : launch_chain(hllc_stream_kernel<2, 0>, grid, block, 0, s, p, rows);
}

// Whether the streaming kernel takes this domain. A warp walks its rows one after another,
// and a small domain has too few warps to hide that; on a narrow one the strips at the west
// and east edge, which check bounds, are too many (us per step, tiles / streaming -- fast dam
// breaks: 1024^2 65.6 / 67.4, 1200^2 87.8 / 82.7, 2048^2 265 / 178; exact lakes: 1024^2 87 /
// 100, 1200^2 116 / 122, 1448^2 164 / 157, 2600 x 800 161 / 163, 1600^2 198 / 185; exact
// dam break, 2048^2 306 / 246). The limits lie above the largest domain on which the tiles
// won (fast 1024^2; exact 2600 x 800, 2.08 M cells) and not at the crossover of square ones,
// which is lower: a fast 1200^2 and an exact 1448^2 would gain 6 % and 4 % by streaming.
#if defined(RB_FAST_MATH)
constexpr long long kHllcStreamCells = 1500000;
#else
constexpr long long kHllcStreamCells = 2300000;
#endif
static_assert(kHllcStreamCells > kNoallocCells, "a streamed domain has a ledger slot per strip and chunk");
static bool hllc_stream_takes(const HllcParams& p) {
  if ((long long)p.ny * p.nx < kHllcStreamCells || p.nx < 30 * kHllcStreamCols) return false;
  // a ledger slot (32 x 8 cells) per strip and chunk: all but narrow and flat domains have them
  const int rows = hllc_stream_rows(p.ny, p.nx);
  const long long blocks = (long long)((p.nx + kHllcStreamCols - 1) / kHllcStreamCols) * ((p.ny + rows - 1) / rows);
  if (blocks > (long long)((p.nx + 31) / 32) * ((p.ny + 7) / 8)) return false;
  return (p.ny + rows - 1) / rows <= 65535 && (long long)(rows + 16) * p.nx < (1LL << 31);
}

#if !defined(RB_FAST_MATH)
// The larger domains of an ensemble in one launch: together they fill the GPU where each
// alone would leave part of its last wave, or all of it, idle (a mix of 20 domains of 128^2
// to 1364^2, us per step: 545 with a launch for each of the three largest and a work-list of
// tiles for the rest, 460 with a launch per scheme and stage).
template <int STAGE, int SRC>
__global__ void __launch_bounds__(32, kHllcStreamWarps)
    ens_hllc_stream_kernel(const __grid_constant__ StreamGroup<HllcParams> g) {
  __shared__ HllcRing<STAGE, SRC> ring;
  pdl_wait();
  int d = 0;
  while ((int)blockIdx.x >= g.first[d + 1]) d++;
  const HllcParams& p = g.p[d];
  const int strips = (p.nx + kHllcStreamCols - 1) / kHllcStreamCols;
  const int b = blockIdx.x - g.first[d];
  hllc_stream_block<STAGE, SRC>(p, b % strips, b / strips, (p.ny + g.rows - 1) / g.rows, (size_t)b, g.rows, ring);
}

constexpr int kEnsHllcMinRows = 11;  // 26 x 11 cells a block: what the ledger's slots allow
bool ens_hllc_stream_fits(const HllcParams& p) {
  const long long blocks = (long long)((p.nx + kHllcStreamCols - 1) / kHllcStreamCols) *
                           ((p.ny + kEnsHllcMinRows - 1) / kEnsHllcMinRows);
  return blocks <= (long long)((p.nx + 31) / 32) * ((p.ny + 7) / 8) && (48 + 16LL) * p.nx < (1LL << 31) &&
         blocks < (1LL << 31) / kStreamGroup;
}

cudaError_t ens_hllc_stream_launch(const HllcParams* p, int n, int stage, cudaStream_t s) {
  const int groups = (n + kStreamGroup - 1) / kStreamGroup;
  for (int k = 0; k < groups; k++) {
    const int d0 = (int)((long long)n * k / groups), m = (int)((long long)n * (k + 1) / groups) - d0;
    StreamGroup<HllcParams> g{};
    long long strip_rows = 0;
    bool src = false;
    for (int d = 0; d < m; d++) {
      const HllcParams& q = g.p[d] = p[d0 + d];
      strip_rows += (long long)((q.nx + kHllcStreamCols - 1) / kHllcStreamCols) * q.ny;
      src |= q.h_comp != nullptr || q.rain_field != nullptr || q.infil != nullptr;
    }
    const long long rows = (strip_rows + 2 * 148 * 16 - 1) / (2 * 148 * 16);
    g.rows = (int)(rows < kEnsHllcMinRows ? kEnsHllcMinRows : (rows > 48 ? 48 : rows));
    for (int d = 0; d < kStreamGroup; d++)
      g.first[d + 1] = g.first[d] + (d < m ? ((g.p[d].nx + kHllcStreamCols - 1) / kHllcStreamCols) *
                                                 ((g.p[d].ny + g.rows - 1) / g.rows)
                                           : 0);
    const dim3 grid(g.first[m]), block(32);
    const cudaError_t e = stage == 1 ? launch_chain(ens_hllc_stream_kernel<1, 0>, grid, block, 0, s, g)
                          : src      ? launch_chain(ens_hllc_stream_kernel<2, 1>, grid, block, 0, s, g)
                                     : launch_chain(ens_hllc_stream_kernel<2, 0>, grid, block, 0, s, g);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
#endif
