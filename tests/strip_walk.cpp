// strip_walk.cpp -- the row-streaming kernels' walk over a chunk, lane by lane on the host.
//
// csrc/li_stream.cuh and csrc/hllc_stream.cuh are compiled as they stand, with the warp's
// exchanges replaced by the lane's own value and the physics by stubs: which words are
// copied, waited for and stored does not depend on either. Every copy has to read inside
// an array of the domain, every cell has to be stored, nothing outside the arrays may be,
// and no copy may still be in flight when a lane leaves its strip.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <deque>
#include <memory>
#include <type_traits>
#include <vector>

#undef __device__
#undef __global__
#undef __shared__
#undef __forceinline__
#undef __launch_bounds__
#undef __grid_constant__
#define __device__
#define __global__
#define __shared__ static
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __grid_constant__
#define RB_FAST_MATH 1

#include "rb_kernels.h"
#include "rbsim.h"

static struct { unsigned x = 0, y = 0; } threadIdx, blockIdx, gridDim;
static long long faults = 0;
static const char* what = "";
static void fault(const char* why) {
  if (faults++ < 20) std::printf("%s: %s\n", what, why);
}

// Arrays of a domain, each between two guards that nothing may touch.
struct Array {
  static constexpr size_t kGuard = 4096;
  std::vector<float> v;
  size_t n;
  explicit Array(size_t n) : v(n + 2 * kGuard, 7.0f), n(n) {}
  float* data() { return v.data() + kGuard; }
  bool holds(const float* p) const { return p >= v.data() + kGuard && p < v.data() + kGuard + n; }
  bool guards_whole() const {
    auto kept = [](float x) { return x == 7.0f; };
    return std::all_of(v.begin(), v.begin() + kGuard, kept) && std::all_of(v.end() - kGuard, v.end(), kept);
  }
};
static std::vector<std::unique_ptr<Array>> arrays;
static float* array(size_t n, float value) {
  arrays.push_back(std::make_unique<Array>(n));
  std::fill_n(arrays.back()->data(), n, value);
  return arrays.back()->data();
}

// Asynchronous copies: words in flight by group, landing when waited for.
struct Word {
  unsigned dst;
  float value;
};
static std::deque<std::vector<Word>> groups;  // the last one is open
static unsigned char* ring_base = nullptr;
static unsigned __cvta_generic_to_shared(const float* p) { return (unsigned)((const unsigned char*)p - ring_base); }

namespace rb {
constexpr float kG = 9.81f, kHDry = 1.0e-3f;
constexpr unsigned kFullWarp = 0xffffffffu;
template <int K, bool CHECK>
void copy_word(unsigned dst, const float* src, bool ok, const float*) {
  if (groups.empty()) groups.emplace_back();
  float value = 0.0f;
  if (!CHECK || ok) {
    const bool inside = std::any_of(arrays.begin(), arrays.end(), [&](const auto& a) { return a->holds(src); });
    if (inside) value = *src;
    else fault("a copy reads outside the domain's arrays");
  }
  groups.back().push_back({dst + K * 128, value});
}
void cp_async_commit() { groups.emplace_back(); }
template <int N>
void cp_async_wait() {  // all but the last N committed groups have landed
  while ((int)groups.size() > N + 1) {
    for (const Word& w : groups.front()) std::memcpy(ring_base + w.dst, &w.value, sizeof w.value);
    groups.pop_front();
  }
}
static void lane_done() {
  for (const auto& g : groups)
    if (!g.empty()) fault("a copy is still in flight when the strip is left");
  groups.clear();
}

int __any_sync(unsigned, bool p) { return p; }
unsigned __ballot_sync(unsigned, bool p) { return p ? kFullWarp : 0u; }
float west_of(float x) { return x; }
float east_of(float x) { return x; }
using std::max;
using std::min;
float rmax(float a, float b) { return a > b ? a : b; }
float rmin(float a, float b) { return a < b ? a : b; }
float rclamp(float x, float lo, float hi) { return rmin(rmax(lo, x), hi); }
void kahan_add(float& t, float&, float inc) { t += inc; }
float div_if(bool use, float x, float y) { return use ? x / y : 0.0f; }
float slope_rcp(float dx) { return 1.0f / dx; }
float manning_divide(float num, float, float, float, float, float) { return num; }
float face_capacity(float, float, float, float, float) { return 0.0f; }
float drain(float h, float, float) { return h; }
template <class T>
T warp_sum(T v) { return v; }
float warp_max(float v) { return v; }
unsigned max_key(float) { return 0; }
void atomicMax(unsigned*, unsigned) {}
void ledger_add(double*, double) {}
void flag_error(unsigned*, unsigned) {}
void pdl_trigger() {}
void pdl_wait() {}
template <class... A>
cudaError_t launch_chain(A&&...) { return cudaSuccess; }

struct LiStepScalars {
  int cur, limit;
  float dt, rain_cont, rain32, scale32, dxdt;
};
bool li_scalars(const LiParams&, LiStepScalars& s) {
  s = LiStepScalars{0, 1, 1.0f, 0.0f, 0.0f, 0.0f, 0.1f};
  return true;
}
struct HllcStageScalars {
  int cur, rain_mode;
  float dt, rain32, scale32;
  float stage[4];
  double wt;
};
bool hllc_scalars(const HllcParams& p, HllcStageScalars& s) {
  s = HllcStageScalars{};
  s.rain_mode = p.h_comp != nullptr && p.rain_field == nullptr ? 1 : 0;
  s.dt = 1.0f;
  return true;
}
struct F2 {
  float x, y;
};
struct Cell {
  float h, un, ut, z;
};
struct Rec {
  float eE, zE, nE, tE, eW, zW, nW, tW, sz;
};
float minmod(float, float) { return 0.0f; }
void primitives_near(float, float, float, float& u, float& v, bool&) { u = v = 0.0f; }
void hllc_near2(F2, F2, F2, F2, F2, F2, F2& a, F2& b, F2& c, bool&) { a = b = c = F2{0.0f, 0.0f}; }
template <bool VOTE>
void hllc_friction(float, bool, float, float, float&, float&) {}
template <bool VOTE>
float wave_speed(float, float, float) { return 0.0f; }

#include "li_stream.cuh"
#include "hllc_stream.cuh"

static bool stored(const float* p, size_t n) {
  return std::none_of(p, p + n, [](float x) { return std::isnan(x); });
}
static void end_of_domain(bool all_stored) {
  if (!all_stored) fault("a cell or a face is stored by no strip");
  for (const auto& a : arrays)
    if (!a->guards_whole()) fault("a store lies outside the domain's arrays");
  arrays.clear();
}

template <int SED, int SRC>
static void li_domain(int ny, int nx, int rows) {
  const size_t cells = (size_t)ny * nx, xf = (size_t)ny * (nx + 1), yf = (size_t)(ny + 1) * nx;
  LiParams p{};
  p.ny = ny, p.nx = nx, p.dx32 = 10.0f;
  p.hb[0] = array(cells, 1.0f), p.qxb[0] = array(xf, 0.0f), p.qyb[0] = array(yf, 0.0f);
  p.hb[1] = array(cells, NAN), p.qxb[1] = array(xf, NAN), p.qyb[1] = array(yf, NAN);
  p.z = array(cells, 0.0f), p.n = array(cells, 0.03f);
  if (SRC != kLiSrcNone) p.h_comp = array(cells, 0.0f);
  if (SRC == kLiSrcAny) p.rain_field = array(cells, 0.0f), p.infil = array(cells, 0.0f);
  if (SED != 0) {
    p.d50 = array(cells, 1.0f);
    p.qs_int_x = array(xf, 0.0f), p.qs_comp_x = array(xf, 0.0f);
    p.qs_int_y = array(yf, 0.0f), p.qs_comp_y = array(yf, 0.0f);
  }
  static LiRing<SED, SRC> ring;
  ring_base = reinterpret_cast<unsigned char*>(ring.row);
  const int strips = (nx + kLiStreamCols - 1) / kLiStreamCols, chunks = (ny + rows - 1) / rows;
  for (int order = 0; order < chunks; order++)
    for (int strip = 0; strip < strips; strip++)
      for (threadIdx.x = 0; threadIdx.x < 32; threadIdx.x++) {
        li_stream_block<SED, SRC>(p, strip, order, chunks, 0, rows, ring);
        lane_done();
      }
  end_of_domain(stored(p.hb[1], cells) && stored(p.qxb[1], xf) && stored(p.qyb[1], yf));
}

template <int STAGE, int SRC>
static void hllc_domain(int ny, int nx, int rows) {
  const size_t cells = (size_t)ny * nx;
  HllcParams p{};
  p.ny = ny, p.nx = nx, p.dx32 = 10.0f;
  p.z = array(cells, 0.0f), p.n = array(cells, 0.03f);
  for (int k = 0; k < 2; k++) {
    const float v = k == 0 ? 1.0f : NAN;
    p.hb[k] = array(cells, v), p.hub[k] = array(cells, v), p.hvb[k] = array(cells, v);
  }
  const float u1 = STAGE == 1 ? NAN : 1.0f;
  p.h1 = array(cells, u1), p.hu1 = array(cells, u1), p.hv1 = array(cells, u1);
  if (SRC != 0) p.h_comp = array(cells, 0.0f), p.rain_field = array(cells, 0.0f), p.infil = array(cells, 0.0f);
  static HllcRing<STAGE, SRC> ring;
  ring_base = reinterpret_cast<unsigned char*>(ring.row);
  const int strips = (nx + kHllcStreamCols - 1) / kHllcStreamCols, chunks = (ny + rows - 1) / rows;
  for (int order = 0; order < chunks; order++)
    for (int strip = 0; strip < strips; strip++)
      for (threadIdx.x = 0; threadIdx.x < 32; threadIdx.x++) {
        hllc_stream_block<STAGE, SRC>(p, strip, order, chunks, 0, rows, ring);
        lane_done();
      }
  end_of_domain(STAGE == 1 ? stored(p.h1, cells) && stored(p.hu1, cells) && stored(p.hv1, cells)
                           : stored(p.hb[1], cells) && stored(p.hub[1], cells) && stored(p.hvb[1], cells));
}

static void domains() {
  // one cell; inner strips and chunks on every side of the conditions that choose them
  const int shapes[][3] = {{1, 1, 11}, {1, 300, 12}, {300, 1, 48}, {14, 30, 14}, {40, 85, 12}, {41, 84, 13},
                           {61, 113, 15}, {75, 112, 25}, {47, 79, 11}, {96, 157, 48}};
  for (const auto& s : shapes) {
    char name[64];
    std::snprintf(name, sizeof name, "%d x %d, %d rows a chunk", s[0], s[1], s[2]);
    what = name;
    li_domain<0, kLiSrcNone>(s[0], s[1], s[2]);
    li_domain<0, kLiSrcComp>(s[0], s[1], s[2]);
    li_domain<0, kLiSrcAny>(s[0], s[1], s[2]);
    li_domain<1, kLiSrcAny>(s[0], s[1], s[2]);
    hllc_domain<1, 0>(s[0], s[1], s[2]);
    hllc_domain<2, 0>(s[0], s[1], s[2]);
    hllc_domain<2, 1>(s[0], s[1], s[2]);
  }
}
}  // namespace rb

int main() {
  rb::domains();
  std::printf("faults %lld\n", faults);
  return faults != 0;
}
