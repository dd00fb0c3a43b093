// Screened map evaluation: the box of an image point decided from a cheaper evaluation of
// the same map, with a proof that the map's own arithmetic decides the same.
//
// What the image kernels need of a point is the box its image lies in.  The maps'
// arithmetic (one rounding per operation in the reference's order, or the explicit-FMA
// variant) is fixed by the results that have to match bit for bit, and its FP64
// instructions bound every image kernel: 78 (strict) or 45 (FMA) a Lorenz RK4 step, 64 a
// forced Duffing step, 23 a Verlet step.  Written for the fewest FP64 instructions - the
// step scaled into the variables, every product fused - the same real-number steps take
// 36, 27 and 7.  Both evaluations differ only by their roundings, so a bound E on the
// distance of the two images (screen.cu, computed on the host for every launch from the
// map, the domain and the depth) makes the screened box the exact one whenever the
// screened image keeps E away from every box boundary.  This is a floating-point filter
// (Fortune and Van Wyk, "Efficient exact arithmetic for computational geometry", 1993):
// a point that fails the test is evaluated again with the map's own arithmetic.
//
// The bound holds while the screened trajectory stays inside the limits `lim`, which the
// kernels check at every step (a maximum over the high words: no FP64 instruction).  All
// of it is FP64; nothing is decided in fewer bits than before.
//
// A step function below is one template for two scalar types: double (device, and the
// host test hook) and Bound (screen.cu), whose operations carry a magnitude and a
// rounding-error bound, so that the bound is derived from the very operations that run.
#pragma once

#include <cmath>
#include <cstdint>

#include "device.cuh"

namespace b12g {

constexpr int kScreenCoef = 10;
constexpr int kScreenMaxBits = 18;   // bisections of a dimension the fixed-point test holds

// Everything a screened launch needs, in the map's scaled coordinates X_j = S_j (x_j - shift_j)
struct ScreenArgs {
  int on;                      // 0: the launch runs the map's own arithmetic alone
  float lim[B12G_MAX_DIM];     // limits on |X_j| as the high words of doubles, see screen_track
  double k[kScreenCoef];       // the map's coefficients
  // the start point: fma(g, sR, fma(v, sA, sB)) from the box's index (v = 1 + index 2^-k),
  // or fma(g, sR, fma(centre, sC, sD)) from the box's centre; sP = sD - 3 sR for points
  // given 3 too high
  double sA[B12G_MAX_DIM], sB[B12G_MAX_DIM], sC[B12G_MAX_DIM], sD[B12G_MAX_DIM], sR[B12G_MAX_DIM];
  double sP[B12G_MAX_DIM];
  // the image's box: fma(X, tA, tB) is 1.5 2^20 + (position in boxes), so its high word
  // counts boxes and its low word is the fraction in units of 2^-32
  double tA[B12G_MAX_DIM], tB[B12G_MAX_DIM];
  uint32_t guard[B12G_MAX_DIM];  // the fraction keeps this far from 0 and from 1
  uint32_t bits[B12G_MAX_DIM];   // bisections of the dimension
  double E[B12G_MAX_DIM];        // the bound on |screened image - exact image| (host use)
};

// ---------------------------------------------------------------------------- operations
__host__ __device__ __forceinline__ double sc_fma(double a, double b, double c)
{
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}
__host__ __device__ __forceinline__ double sc_add(double a, double b)
{
#ifdef __CUDA_ARCH__
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}
__host__ __device__ __forceinline__ double sc_mul(double a, double b)
{
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
__host__ __device__ __forceinline__ double sc_neg(double a) { return -a; }
// 2 a + b, a / 2 + b
__host__ __device__ __forceinline__ double sc_fma2(double a, double b) { return sc_fma(2.0, a, b); }
__host__ __device__ __forceinline__ double sc_fma_half(double a, double b) { return sc_fma(0.5, a, b); }
// a value times a coefficient that the scaling makes 1 up to the roundings of the scales
__host__ __device__ __forceinline__ double sc_near(double a) { return a; }

// ---------------------------------------------------------------------------- Lorenz
// X = c (x, y, z - rho) with c = h/2 turns k-scaled stages into bare products:
//   c X0' = s (X1 - X0), c X1' = -X0 X2 - c X1, c X2' = X0 X1 - q X2 - kappa
// with s = c sigma, q = c beta, kappa = c^2 beta rho.  Classical RK4 as
//   a = X + c X'(X), b = X + c X'(a), w = 2 (b + c X'(b) - X) ... :
//   X+ = (a + 2 b + d - X + c X'(d)) / 3 with d = X + 2 c X'(b),
// the first component (linear) summed from its differences instead: 36 operations.
// k: s, -c, 1 - c, -q, 1 - q, -kappa, 2 s, s / 3, 1 / 3, -kappa / 3
template<class T, class K>
__host__ __device__ __forceinline__ void lorenz_screen_step(const K* k, T (&x)[3])
{
  const T d1 = sc_add(x[1], sc_neg(x[0]));
  const T a0 = sc_fma(k[0], d1, x[0]);
  const T a1 = sc_fma(sc_neg(x[0]), x[2], sc_mul(k[2], x[1]));
  const T a2 = sc_fma(x[0], x[1], sc_fma(k[4], x[2], k[5]));
  const T xk = sc_add(x[2], k[5]);
  const T d2 = sc_add(a1, sc_neg(a0));
  const T b0 = sc_fma(k[0], d2, x[0]);
  const T b1 = sc_fma(sc_neg(a0), a2, sc_fma(k[1], a1, x[1]));
  const T b2 = sc_fma(a0, a1, sc_fma(k[3], a2, xk));
  const T d3 = sc_add(b1, sc_neg(b0));
  const T v1 = sc_fma(sc_neg(b0), b2, sc_mul(k[1], b1));
  const T v2 = sc_fma(b0, b1, sc_fma(k[3], b2, k[5]));
  const T c0 = sc_fma(k[6], d3, x[0]);
  const T c1 = sc_fma2(v1, x[1]);
  const T c2 = sc_fma2(v2, x[2]);
  const T d4 = sc_add(c1, sc_neg(c0));
  const T e1 = sc_fma2(sc_add(b1, v1), a1);
  const T e2 = sc_fma2(sc_add(b2, v2), a2);
  x[0] = sc_fma(k[7], sc_fma2(sc_add(d2, d3), sc_add(d1, d4)), x[0]);
  x[1] = sc_mul(k[8], sc_fma(sc_neg(c0), c2, sc_fma(k[1], c1, e1)));
  x[2] = sc_fma(k[8], sc_fma(c0, c1, sc_fma(k[3], c2, e2)), k[9]);
}

// ---------------------------------------------------------------------------- coupled Duffing
// Stormer-Verlet of H = |p|^2/2 - q1^2/2 + q1^4/4 + 1.69 q2^2/2 + 0.1 q1^2 q2^2 with
// Q1 = h q1, Q2 = sqrt(0.2) h q2, P1 = h^2 p1, P2 = sqrt(0.2) h^2 p2: a drift is Q + P and a
// kick P1 += Q1 (h^2 - Q1^2 - Q2^2), P2 += Q2 (-1.69 h^2 - 0.2 Q1^2).  The half drifts of
// consecutive steps join: 7 operations a step.  These steps alone took the
// image launches of the depth-24 continuation from 15.5 to 11.0 ms; the Philox points and the
// marking are most of what is left.
// k: h^2, 0.2, -(1.69 + 0.2) h^2
template<class T, class K>
__host__ __device__ __forceinline__ void duffing_screen_kick(const K* k, T (&x)[4])
{
  const T t = sc_fma(sc_neg(x[0]), x[0], k[0]);
  const T u = sc_fma(sc_neg(x[1]), sc_near(x[1]), t);
  const T s = sc_fma(k[1], t, k[2]);
  x[2] = sc_fma(sc_near(x[0]), u, x[2]);
  x[3] = sc_fma(sc_near(x[1]), s, x[3]);
}
template<class T>
__host__ __device__ __forceinline__ void duffing_screen_drift(T (&x)[4])
{
  x[0] = sc_add(x[0], sc_near(x[2]));
  x[1] = sc_add(x[1], sc_near(x[3]));
}
template<class T>
__host__ __device__ __forceinline__ void duffing_screen_half_drift(T (&x)[4])
{
  x[0] = sc_fma_half(sc_near(x[2]), x[0]);
  x[1] = sc_fma_half(sc_near(x[3]), x[1]);
}

// ---------------------------------------------------------------------------- forced Duffing
// x'' + delta x' + alpha x + beta x^3 = gamma cos t (beta > 0) with c = h/2,
// X = c sqrt(beta) x and V = c^2 sqrt(beta) x': c X' = V and
//   c V' = -c delta V - X (c^2 alpha + X^2) + F(t),
// RK4 put together as for Lorenz: 25 operations a step and the two of F = k[3] cos at the
// middle and the end.  f0, f1, f2: F at the stages' times.  These steps
// alone took the image launches of a depth-19 job from 3.85 to 2.03 ms, of a depth-22 one from
// 5.44 to 2.72 (0.80 and 1.40 with the work queue of 32-point units: small launches).
// k: -c^2 alpha, -c delta, 1 - c delta, c^3 sqrt(beta) gamma, 1 / 3
template<class T, class K>
__host__ __device__ __forceinline__ void forced_screen_step(const K* k, const T& f0, const T& f1, const T& f2,
                                                            T (&x)[2])
{
  const T a0 = sc_add(x[0], sc_near(x[1]));
  const T a1 = sc_fma(x[0], sc_fma(sc_neg(x[0]), sc_near(x[0]), k[0]), sc_fma(k[2], x[1], f0));
  const T b0 = sc_add(x[0], sc_near(a1));
  const T b1 = sc_fma(a0, sc_fma(sc_neg(a0), sc_near(a0), k[0]), sc_fma(k[1], a1, sc_add(x[1], f1)));
  const T v1 = sc_fma(b0, sc_fma(sc_neg(b0), sc_near(b0), k[0]), sc_fma(k[1], b1, f1));
  const T d0 = sc_fma2(sc_near(b1), x[0]);
  const T d1 = sc_fma2(v1, x[1]);
  const T e1 = sc_add(sc_fma2(sc_add(b1, v1), a1), f2);
  x[0] = sc_fma(k[4], sc_near(sc_fma2(sc_add(a1, b1), sc_add(x[1], d1))), x[0]);
  x[1] = sc_mul(k[4], sc_fma(d0, sc_fma(sc_neg(d0), sc_near(d0), k[0]), sc_fma(k[1], d1, e1)));
}

// ---------------------------------------------------------------------------- tracking
#ifdef __CUDACC__
// m = max(m, |x|) on the high words of doubles read as floats, which order like the
// doubles; a NaN (as a float: any double of at least 2^1017, an infinity or a NaN) stays
__device__ __forceinline__ void screen_track(float& m, double x)
{
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(m) : "f"(fabsf(__int_as_float(__double2hiint(x)))));
}
// of two values in one instruction
__device__ __forceinline__ float screen_high(double x) { return __int_as_float(__double2hiint(x)); }
__device__ __forceinline__ void screen_track2(float& m, float x, float y)
{
  asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(x), "f"(y));
}
#endif

// maps with a screened evaluation: run() advances X over the map's steps and returns
// whether the trajectory kept within the limits
template<class Map> struct Screen { static constexpr bool kOk = false; };

#ifdef __CUDACC__
template<class A> struct Screen<LorenzMap<A>> {
  static constexpr bool kOk = true;
  static constexpr int kOwnCount = 2;                     // rho: kappa and kappa / 3
  static __host__ __device__ constexpr int own(int i) { return i == 0 ? 5 : 9; }
  static __device__ __forceinline__ bool run(const ScreenArgs& s, const MapParams& map, double (&x)[3])
  {
    return run(s.k, s.lim, map, x);
  }
  static __device__ __forceinline__ bool run(const double* k, const float* lim, const MapParams& map, double (&x)[3])
  {
    float m0 = 0.f, m1 = 0.f, m2 = 0.f;
    if (map.steps & 1u) {
      screen_track(m0, x[0]);
      screen_track(m1, x[1]);
      screen_track(m2, x[2]);
      lorenz_screen_step(k, x);
    }
    // twenty steps a trip (the usual number): the coefficients are loaded once for them
#pragma unroll 10
    for (uint32_t i = map.steps >> 1; i > 0; --i) {
      const float h0 = screen_high(x[0]), h1 = screen_high(x[1]), h2 = screen_high(x[2]);
      lorenz_screen_step(k, x);
      screen_track2(m0, h0, screen_high(x[0]));
      screen_track2(m1, h1, screen_high(x[1]));
      screen_track2(m2, h2, screen_high(x[2]));
      lorenz_screen_step(k, x);
    }
    return m0 <= lim[0] && m1 <= lim[1] && m2 <= lim[2];
  }
};

template<> struct Screen<CoupledDuffingMap> {
  static constexpr bool kOk = true;
  // the limits hold for the positions at every kick and for the first momenta
  static __device__ __forceinline__ bool run(const ScreenArgs& s, const MapParams& map, double (&x)[4])
  {
    float m0 = 0.f, m1 = 0.f, m2 = 0.f, m3 = 0.f;
    screen_track(m2, x[2]);
    screen_track(m3, x[3]);
    duffing_screen_half_drift(x);
    auto kick = [&]() {
      screen_track(m0, x[0]);
      screen_track(m1, x[1]);
      duffing_screen_kick(s.k, x);
    };
#pragma unroll 9
    for (uint32_t i = 1; i < map.steps; ++i) {
      kick();
      duffing_screen_drift(x);
    }
    kick();
    duffing_screen_half_drift(x);
    return m0 <= s.lim[0] && m1 <= s.lim[1] && m2 <= s.lim[2] && m3 <= s.lim[3];
  }
};

template<> struct Screen<ForcedDuffingMap> {
  static constexpr bool kOk = true;
  static constexpr int kOwnCount = 1;                     // gamma: the scale of F
  static __host__ __device__ constexpr int own(int) { return 3; }
  static __device__ __forceinline__ bool run(const ScreenArgs& s, const MapParams& map, double (&x)[2])
  {
    return run(s.k, s.lim, map, x);
  }
  static __device__ __forceinline__ bool run(const double* k, const float* lim, const MapParams& map, double (&x)[2])
  {
    float m0 = 0.f, m1 = 0.f;
    double f0 = __dmul_rn(k[3], __ldg(map.table));
    const double* tab = map.table;
    auto step = [&]() {
      const double f1 = __dmul_rn(k[3], __ldg(tab + 1));
      const double f2 = __dmul_rn(k[3], __ldg(tab + 2));
      forced_screen_step(k, f0, f1, f2, x);
      f0 = f2;
      tab += 2;
    };
    if (map.steps & 1u) {
      screen_track(m0, x[0]);
      screen_track(m1, x[1]);
      step();
    }
#pragma unroll 1
    for (uint32_t i = map.steps >> 1; i > 0; --i) {
      const float h0 = screen_high(x[0]), h1 = screen_high(x[1]);
      step();
      screen_track2(m0, h0, screen_high(x[0]));
      screen_track2(m1, h1, screen_high(x[1]));
      step();
    }
    return m0 <= lim[0] && m1 <= lim[1];
  }
};

// Whether a warp tries the screened evaluation on its next piece of work.  A warp with an
// undecided point runs both evaluations, so where many points stay undecided (trajectories
// that leave the limits, in domains or maps whose bound leaves no room for wider ones) trying
// costs more than it saves.  After two pieces in a row in which some lane had half of its
// points undecided the warp takes the map's own arithmetic for the next 3 pieces, and after
// another one, or more, for 31.  Two, since 4 % of the points are undecided in the usual
// forced Duffing jobs, where trying still pays.  Counted by pieces, not by points, since the
// points' loop is bound by its instructions (a vote for every 32 points cost a Lorenz job of
// depth 27 1.2 %), but in a tree's two-dimensional image launches, whose points are longer and
// launches smaller, by units of 32 points (a forced Duffing job of depth 19: 1,142 us, by
// pieces 1,222, always trying 1,174; the batches' launches lose 1 to 2 % either way).
// Images of 250,000 Lorenz boxes (125 points, h = 0.02, radius 10 around 0; 3 % of the points
// decided): 2.92 ms (strict) and 1.86 (FMA), always trying 4.21 and 3.17, never 2.82 and 1.75.
// `undecided`: the lane's undecided points of the piece's `tries`.  Every lane calls note()
// after every piece.
struct ScreenTrial {
  uint32_t skip = 0, failed = 0;
  static __host__ __device__ constexpr bool by_unit(int dim) { return dim == 2; }
  __device__ __forceinline__ bool on() const { return skip == 0; }
  __device__ __forceinline__ void note(uint32_t undecided, uint32_t tries)
  {
    if (skip) {
      --skip;
      return;
    }
    const bool bad = __any_sync(0xFFFFFFFFu, undecided != 0 && 2u * undecided >= tries);
    failed = bad ? min(failed + 1u, 3u) : 0u;
    skip = failed < 2u ? 0u : failed == 2u ? 3u : 31u;
  }
};

// the double 1 + index 2^-k (exact for k <= 20)
__device__ __forceinline__ double screen_index(uint32_t index, uint32_t k)
{
  return __hiloint2double(int(0x3FF00000u | (index << (20u - k))), 0);
}

// The box of the screened image X: its per-dimension indices in `bits` and whether it lies
// in the domain; returns whether the exact evaluation is certain to decide the same.  A
// position outside the range of the fixed-point form (or a box outside the domain) has a
// high word outside [0, 2^k), compared unsigned.
template<int D>
__device__ __forceinline__ bool screen_locate(const ScreenArgs& s, const double (&x)[D], uint32_t (&bits)[D],
                                              bool& inside)
{
  bool sure = true;
  inside = true;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    const double t = __fma_rn(x[j], s.tA[j], s.tB[j]);
    const uint32_t b = uint32_t(__double2hiint(t)) - 0x41380000u;
    sure = sure && uint32_t(__double2loint(t)) - s.guard[j] <= ~(2u * s.guard[j]);
    inside = inside && (b >> s.bits[j]) == 0u;
    bits[j] = b;
  }
  return sure;
}
#endif

// One instance's part of a batched launch (batch.cu): the start, position and limits of its
// parameters at its depth.  The coefficients are the launch's (BatchArgs::sk) but for the
// instance's own: coefficient Screen<Map>::own(i) is own[i], i < Screen<Map>::kOwnCount.
struct alignas(16) ScreenRec {
  double sB[3], tB[3], sR[3], tA[3];
  double own[2];
  uint32_t guard[3];
  float lim[3];
  uint32_t k;                  // bisections of the dimensions, a byte each
  uint32_t on;
};

// ---------------------------------------------------------------------------- host
// a map's part of a screen over one box of states: scales, shifts, limits and the distance
// E of the two images
struct MapBound {
  double scale[B12G_MAX_DIM] = {1.0, 1.0, 1.0, 1.0}, shift[B12G_MAX_DIM] = {0.0, 0.0, 0.0, 0.0};
  double lim[B12G_MAX_DIM] = {0.0, 0.0, 0.0, 0.0};   // unscaled, around the shift
  double E[B12G_MAX_DIM] = {0.0, 0.0, 0.0, 0.0};
};

// The depth-independent part of a screen: a map's bounds over multiples of the domain (found
// when a depth first asks for them) and its coefficients.
constexpr int kScreenBoxes = 7;
struct ScreenPlan {
  uint32_t kind = 0;
  MapParams map{};
  Domain dom{};
  int dim = 0;
  double gmax = 0.0;
  bool possible = false;
  bool wide = false;           // box 0 goes beyond the others
  bool found[kScreenBoxes] = {};
  MapBound bound[kScreenBoxes];
  double k[kScreenCoef] = {};
};
// grid points at most gmax box radii from the centre
ScreenPlan screen_plan(uint32_t map_kind, const MapParams& map, const Domain& dom, int dim, double gmax);
// fills `s` for launches over boxes of `depth`; s.on tells whether the screened evaluation
// applies (screen.cu states when)
void screen_at(ScreenPlan& plan, int depth, ScreenArgs& s);
// both at once; plan: null, or one kept for launches in this domain, made again when the map
// or the reach is another (a tree's: its launches are not called from several threads)
void fill_screen(uint32_t map_kind, const MapParams& map, const Domain& dom, int dim, int depth, double gmax,
                 ScreenPlan* plan, ScreenArgs& s);
// the largest |coordinate| of a grid's points
double grid_reach(uint32_t grid_kind, const GridParams& g);
// the record of a batched instance; false where it cannot share `common`'s coefficients and
// scales (common.on == 0: the first one, which sets them)
bool screen_record(uint32_t map_kind, int dim, const ScreenArgs& s, ScreenArgs& common, ScreenRec& rec);
// whether a batched launch of `all` instances (or boxes) runs screened when the bound covers
// `on` of them
inline bool screen_covers(uint64_t on, uint64_t all) { return on > 0 && 2 * on >= all; }

}  // namespace b12g
