// Host side of the screened map evaluation (screen.cuh): the scaled coefficients and the
// bound on the distance between the screened image and the map's own.
//
// With u = 2^-53 and Phi the real-number step with the given double parameters, both
// evaluations are Phi plus local roundings.  If every screened state lies in the box
// |X_j| <= lim_j and the two trajectories are within eta = 2^-20 lim of each other, then
//   |x^ - x~|_(n+1) <= G |x^ - x~|_n + d^ + d~   (component by component),
// G a bound on |D Phi| over the box grown by eta, d^ and d~ bounds on the local roundings
// of one step there.  All three come from running the step's operations on `Bound`: a
// magnitude, the accumulated rounding error and the magnitudes of the derivatives by the
// step's inputs.  Iterated over the map's steps from the start points' distance this gives
// E; eta is checked at the end.  Only |x^ - x~| <= E matters, not the integrator's own
// error, so E stays near the roundings times the flow's growth: for the benchmark's Lorenz
// map over twice its domain 4e-6, against boxes 0.12 wide at depth 27 and distances seen of
// 3e-14.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "kernels.h"
#include "screen.cuh"
#include "tree.h"

namespace b12g {

namespace {

constexpr double kU = 0x1p-53;
constexpr double kEta = 0x1p-20;

struct Bound {
  double m = 0.0;              // magnitude of the exact value
  double e = 0.0;              // of (computed - exact)
  double d[B12G_MAX_DIM] = {0.0, 0.0, 0.0, 0.0};   // of the derivatives by the inputs
};

__host__ __device__ Bound rounded(Bound r)
{
  r.e += kU * (r.m + r.e);
  return r;
}

// a rounded constant (error at most `ulps` units of 2^-53 relative)
__host__ __device__ Bound constant(double v, double ulps)
{
  Bound b;
  b.m = v < 0.0 ? -v : v;
  b.e = ulps * kU * b.m;
  return b;
}

__host__ __device__ Bound product(const Bound& a, const Bound& b)
{
  Bound r;
  r.m = a.m * b.m;
  r.e = a.e * b.m + a.m * b.e + a.e * b.e;
  for (int j = 0; j < B12G_MAX_DIM; ++j) r.d[j] = a.d[j] * b.m + a.m * b.d[j];
  return r;
}

__host__ __device__ Bound sum(const Bound& a, const Bound& b)
{
  Bound r;
  r.m = a.m + b.m;
  r.e = a.e + b.e;
  for (int j = 0; j < B12G_MAX_DIM; ++j) r.d[j] = a.d[j] + b.d[j];
  return r;
}

__host__ __device__ Bound sc_fma(const Bound& a, const Bound& b, const Bound& c) { return rounded(sum(product(a, b), c)); }
__host__ __device__ Bound sc_add(const Bound& a, const Bound& b) { return rounded(sum(a, b)); }
__host__ __device__ Bound sc_mul(const Bound& a, const Bound& b) { return rounded(product(a, b)); }
__host__ __device__ Bound sc_neg(const Bound& a) { return a; }
__host__ __device__ Bound sc_fma2(const Bound& a, const Bound& b) { return rounded(sum(product(constant(2.0, 0.0), a), b)); }
__host__ __device__ Bound sc_fma_half(const Bound& a, const Bound& b) { return rounded(sum(product(constant(0.5, 0.0), a), b)); }
__host__ __device__ Bound sc_near(Bound a)
{
  a.e += 16.0 * kU * a.m;
  return a;
}

// |x_(n+1) - y_(n+1)| <= G |x_n - y_n| + d
struct StepBound {
  double G[B12G_MAX_DIM][B12G_MAX_DIM];
  double d[B12G_MAX_DIM];
};

void identity_box(const double* lim, int dim, Bound* x)
{
  for (int j = 0; j < dim; ++j) {
    x[j] = Bound{};
    x[j].m = lim[j] * (1.0 + kEta);
    x[j].d[j] = 1.0;
  }
}

// E from the distance e0 of the start points over `steps` steps
void iterate_bound(const StepBound& b, int dim, uint32_t steps, const double* e0, double* E)
{
  double e[B12G_MAX_DIM];
  for (int j = 0; j < dim; ++j) e[j] = e0[j];
  for (uint32_t n = 0; n < steps; ++n) {
    double f[B12G_MAX_DIM], most = 0.0;
    for (int i = 0; i < dim; ++i) {
      f[i] = b.d[i];
      for (int j = 0; j < dim; ++j) f[i] += b.G[i][j] * e[j];
      most = std::max(most, f[i]);
    }
    for (int i = 0; i < dim; ++i) e[i] = f[i];
    if (!(most < 1e300)) break;
  }
  for (int j = 0; j < dim; ++j) E[j] = e[j] * (1.0 + 0x1p-20);
}

// ---- Lorenz: classical RK4 in the map's order (Map_Lorenz.h:10-44, MapTools.hpp:118-182).
// Inputs (x, y, z - rho); the derivative of rho x - y - x z is that of -x (z - rho) - y.
// The explicit-FMA variant makes a subset of these roundings.
void lorenz_rhs(const Bound* a, double sigma, double rho, double beta, Bound* r)
{
  Bound z = a[2];
  z.m += std::fabs(rho);
  r[0] = sc_mul(constant(sigma, 0.0), sc_add(a[1], a[0]));
  const Bound exact = sum(product(a[0], a[2]), a[1]);
  const Bound done = sc_add(sc_add(sc_mul(constant(rho, 0.0), a[0]), a[1]), sc_mul(a[0], z));
  r[1] = exact;
  r[1].e = done.e;
  r[2] = sc_add(sc_mul(constant(beta, 0.0), z), sc_mul(a[0], a[1]));
}

// b + c k, the third component carrying rho
void lorenz_madd(const Bound* k, const Bound& c, const Bound* b, double rho, Bound* out)
{
  for (int j = 0; j < 3; ++j) {
    Bound r = sum(sc_mul(c, k[j]), b[j]);
    r.e += kU * (r.m + r.e + (j == 2 ? std::fabs(rho) : 0.0));
    out[j] = r;
  }
}

void lorenz_coef(double h, double sigma, double rho, double beta, double* k)
{
  const double c = h / 2.0, q = c * beta, kappa = c * c * beta * rho;
  const double v[kScreenCoef] = {c * sigma, -c, 1.0 - c, -q, 1.0 - q, -kappa, 2.0 * c * sigma, c * sigma / 3.0,
                                 1.0 / 3.0, -kappa / 3.0};
  for (int i = 0; i < kScreenCoef; ++i) k[i] = v[i];
}

void lorenz_bound(const MapParams& map, const double* lim, const double* e0, MapBound& b, double* coef)
{
  const double h = map.h, sigma = map.p[0], rho = map.p[1], beta = map.p[2], c = h / 2.0;
  for (int j = 0; j < 3; ++j) {
    b.scale[j] = c;
    b.shift[j] = j == 2 ? rho : 0.0;
    b.lim[j] = lim[j];
  }
  lorenz_coef(h, sigma, rho, beta, coef);
  StepBound s;
  Bound x[3], k[3], a[3], res[3];
  identity_box(b.lim, 3, x);
  lorenz_rhs(x, sigma, rho, beta, k);
  lorenz_madd(k, constant(h / 6.0, 1.0), x, rho, res);
  lorenz_madd(k, constant(c, 0.0), x, rho, a);
  lorenz_rhs(a, sigma, rho, beta, k);
  lorenz_madd(k, constant(h / 3.0, 1.0), res, rho, res);
  lorenz_madd(k, constant(c, 0.0), x, rho, a);
  lorenz_rhs(a, sigma, rho, beta, k);
  lorenz_madd(k, constant(h / 3.0, 1.0), res, rho, res);
  lorenz_madd(k, constant(h, 0.0), x, rho, a);
  lorenz_rhs(a, sigma, rho, beta, k);
  lorenz_madd(k, constant(h / 6.0, 1.0), res, rho, res);
  // the screened step in its scaled coordinates (1 - c and 1 - q: the rounding of the
  // difference and that of q)
  Bound kb[kScreenCoef], sx[3];
  for (int i = 0; i < kScreenCoef; ++i) kb[i] = constant(coef[i], 8.0);
  kb[2].e = kb[4].e = 8.0 * kU * (1.0 + std::fabs(c) + std::fabs(coef[3]));
  for (int j = 0; j < 3; ++j) sx[j].m = x[j].m * std::fabs(c);
  lorenz_screen_step(kb, sx);
  for (int i = 0; i < 3; ++i) {
    for (int j = 0; j < 3; ++j) s.G[i][j] = res[i].d[j];
    s.d[i] = res[i].e + sx[i].e / std::fabs(c);
  }
  iterate_bound(s, 3, map.steps, e0, b.E);
}

// ---- coupled Duffing: Stormer-Verlet in the map's order (MapTools.hpp:371-421).  The
// limits hold for the positions at the kicks and the first momenta; the momenta then grow by
// at most |h| max |force| a step, and the positions between the kicks differ from those at
// them by half a drift.
const double kDuffingStiff = 1.69, kDuffingCouple = 0.2;

void cap(Bound& x, double m) { x.m = std::min(x.m, m); }

void coupled_bound(const MapParams& map, const double* lim, const double* e0, MapBound& b, double* coef)
{
  const double h = map.h, ah = std::fabs(h), root = std::sqrt(kDuffingCouple);
  double q[2], grown[4];
  for (int j = 0; j < 4; ++j) b.lim[j] = lim[j];
  for (int j = 0; j < 2; ++j) q[j] = b.lim[j] * (1.0 + kEta);
  const double f[2] = {q[0] + q[0] * q[0] * q[0] + kDuffingCouple * q[0] * q[1] * q[1],
                       kDuffingStiff * q[1] + kDuffingCouple * q[0] * q[0] * q[1]};
  for (int j = 0; j < 2; ++j) {
    grown[2 + j] = (b.lim[2 + j] + double(map.steps) * ah * f[j]) * (1.0 + kEta);
    grown[j] = q[j] + 0.5 * ah * grown[2 + j] * (1.0 + kEta);
    b.scale[j] = j == 0 ? h : root * h;
    b.scale[2 + j] = j == 0 ? h * h : root * h * h;
  }
  coef[0] = h * h;
  coef[1] = kDuffingCouple;
  coef[2] = -(kDuffingStiff + kDuffingCouple) * h * h;
  StepBound s;
  Bound x[4];
  identity_box(grown, 4, x);
  auto half_drift = [&]() {
    for (int j = 0; j < 2; ++j)
      x[j] = sc_add(x[j], sc_mul(sc_mul(constant(0.5, 0.0), x[2 + j]), constant(h, 0.0)));
  };
  half_drift();
  for (int j = 0; j < 2; ++j) cap(x[j], q[j]);
  const Bound couple = constant(kDuffingCouple, 0.0);
  const Bound f0 = sc_add(sc_add(x[0], sc_mul(sc_mul(x[0], x[0]), x[0])), sc_mul(sc_mul(sc_mul(couple, x[0]), x[1]), x[1]));
  const Bound f1 = sc_add(sc_mul(constant(kDuffingStiff, 0.0), x[1]), sc_mul(sc_mul(sc_mul(couple, x[0]), x[0]), x[1]));
  x[2] = sc_add(x[2], sc_mul(f0, constant(h, 0.0)));
  x[3] = sc_add(x[3], sc_mul(f1, constant(h, 0.0)));
  half_drift();
  // the screened step with both its half drifts (joined, they make fewer roundings)
  Bound sx[4], k[3];
  for (int i = 0; i < 3; ++i) k[i] = constant(coef[i], i == 1 ? 0.0 : 8.0);
  for (int j = 0; j < 4; ++j) sx[j].m = grown[j] * (1.0 + kEta) * std::fabs(b.scale[j]) * (1.0 + kEta);
  duffing_screen_half_drift(sx);
  for (int j = 0; j < 2; ++j) cap(sx[j], q[j] * std::fabs(b.scale[j]) * (1.0 + kEta));
  duffing_screen_kick(k, sx);
  duffing_screen_half_drift(sx);
  for (int i = 0; i < 4; ++i) {
    for (int j = 0; j < 4; ++j) s.G[i][j] = x[i].d[j];
    s.d[i] = x[i].e + sx[i].e / std::fabs(b.scale[i]) * (1.0 + kEta);
  }
  iterate_bound(s, 4, map.steps, e0, b.E);
}

// ---- forced Duffing: classical RK4 of (x, v) in the map's order.  Over a period of 200
// steps the component-wise bound, blind to the rotation of the flow, would grow by e^20;
// here the distance is bounded in the norm |(w x, v)|_2.  With J the Jacobian of the right
// hand side in that norm, mu >= the largest eigenvalue of its symmetric part and L >= |J|_2
// over the stages, D Phi = I + h A + R with A the weighted mean of the stages' Jacobians,
// |I + h A| <= sqrt(1 + 2 h mu + h^2 L^2) and |R| <= (hL)^2/2 + (hL)^3/6 + (hL)^4/24.  w is
// the best of a few.
void forced_rhs(const Bound* a, const double* p, Bound* r)
{
  r[0] = a[1];
  r[1] = sc_add(sc_add(sc_add(sc_mul(constant(p[0], 0.0), a[1]), sc_mul(constant(p[1], 0.0), a[0])),
                       sc_mul(constant(p[2], 0.0), sc_mul(sc_mul(a[0], a[0]), a[0]))),
                constant(p[3], 1.0));                    // gamma cos: |cos| <= 1, one rounding
}

void forced_madd(const Bound* k, const Bound& c, const Bound* b, Bound* out)
{
  for (int j = 0; j < 2; ++j) out[j] = sc_add(sc_mul(c, k[j]), b[j]);
}

void forced_bound(const MapParams& map, const double* lim, const double* e0, MapBound& b, double* coef)
{
  const double h = map.h, c = h / 2.0, delta = map.p[0], alpha = map.p[1], beta = map.p[2], root = std::sqrt(beta);
  b.scale[0] = c * root;
  b.scale[1] = c * c * root;
  for (int j = 0; j < 2; ++j) b.lim[j] = lim[j];
  const double v[5] = {-c * c * alpha, -c * delta, 1.0 - c * delta, c * c * c * root * map.p[3], 1.0 / 3.0};
  for (int i = 0; i < 5; ++i) coef[i] = v[i];
  Bound x[2], k[2], a[2], res[2];
  identity_box(b.lim, 2, x);
  double sx = x[0].m;
  forced_rhs(x, map.p, k);
  forced_madd(k, constant(h / 6.0, 1.0), x, res);
  forced_madd(k, constant(c, 0.0), x, a);
  sx = std::max(sx, a[0].m);
  forced_rhs(a, map.p, k);
  forced_madd(k, constant(h / 3.0, 1.0), res, res);
  forced_madd(k, constant(c, 0.0), x, a);
  sx = std::max(sx, a[0].m);
  forced_rhs(a, map.p, k);
  forced_madd(k, constant(h / 3.0, 1.0), res, res);
  forced_madd(k, constant(h, 0.0), x, a);
  sx = std::max(sx, a[0].m);
  forced_rhs(a, map.p, k);
  forced_madd(k, constant(h / 6.0, 1.0), res, res);
  // the screened step
  Bound kb[5], sxv[2];
  for (int i = 0; i < 5; ++i) kb[i] = constant(coef[i], 8.0);
  kb[2].e = 8.0 * kU * (1.0 + std::fabs(c * delta));
  for (int j = 0; j < 2; ++j) sxv[j].m = x[j].m * b.scale[j] * (1.0 + kEta);
  const Bound f = sc_mul(kb[3], constant(1.0, 0.0));
  forced_screen_step(kb, f, f, f, sxv);
  double d[2];
  for (int j = 0; j < 2; ++j) d[j] = res[j].e + sxv[j].e / b.scale[j] * (1.0 + kEta);
  // -alpha - 3 beta x^2 over |x| <= sx lies between these
  const double g0 = -alpha, g1 = -alpha - 3.0 * beta * sx * sx, gm = std::max(std::fabs(g0), std::fabs(g1));
  double best = INFINITY, bw = 1.0;
  for (int i = -8; i <= 24; ++i) {
    const double w = std::exp2(0.25 * i);
    const double q = 0.5 * std::max(std::fabs(w + g0 / w), std::fabs(w + g1 / w));
    const double mu = 0.5 * (-delta + std::sqrt(delta * delta + 4.0 * q * q));
    const double ad = std::fabs(delta);
    const double L = std::sqrt(std::max(gm / w, w + ad) * std::max(w, gm / w + ad)), hl = h * L;
    const double grow = std::sqrt(std::max(0.0, 1.0 + 2.0 * h * mu + hl * hl)) +
                        hl * hl * (0.5 + hl * (1.0 / 6.0 + hl / 24.0));
    if (grow < best) { best = grow; bw = w; }
  }
  best *= 1.0 + 0x1p-40;
  const double step = std::hypot(bw * d[0], d[1]);
  double e = std::hypot(bw * e0[0], e0[1]);
  for (uint32_t n = 0; n < map.steps && e < 1e300; ++n) e = best * e + step;
  e *= 1.0 + 0x1p-20;
  b.E[0] = e / bw;
  b.E[1] = e;
}

// magnitudes for which no product or scale below leaves the normal range
bool moderate(double v) { return std::fabs(v) <= 0x1p40; }
bool moderate_nonzero(double v) { return std::fabs(v) >= 0x1p-40 && std::fabs(v) <= 0x1p40; }

}  // namespace

double grid_reach(uint32_t grid_kind, const GridParams& g)
{
  if (grid_kind == B12G_GRID_PHILOX) return 1.0;
  double m = 0.0;
  for (uint32_t i = 0; i < g.n; ++i) m = std::max(m, std::fabs(g.coord[i]));
  return grid_kind == B12G_GRID_FULL ? m * std::fabs(g.eps1) : m;
}

ScreenPlan screen_plan(uint32_t map_kind, const MapParams& map, const Domain& dom, int dim, double gmax)
{
  ScreenPlan p;
  p.kind = map_kind;
  p.map = map;
  p.dom = dom;
  p.dim = dim;
  p.gmax = gmax;
  if (map_kind == B12G_MAP_HENON) return p;      // five operations: nothing to save
  if (map.steps == 0 || map.steps > 4096 || !moderate_nonzero(map.h) || !moderate(gmax)) return p;
  for (double v : map.p)
    if (!moderate(v)) return p;
  for (int j = 0; j < dim; ++j)
    if (!moderate_nonzero(dom.r[j]) || !moderate(dom.c[j])) return p;
  if (map_kind == B12G_MAP_FORCED_DUFFING && !(map.h > 0.0 && map.p[2] > 0.0 && moderate_nonzero(map.p[2]))) return p;
  p.possible = true;
  return p;
}

namespace {

// A double whose operations are the plain ones, for estimates
struct Rough {
  double v;
};
Rough sc_fma(Rough a, Rough b, Rough c) { return {a.v * b.v + c.v}; }
Rough sc_add(Rough a, Rough b) { return {a.v + b.v}; }
Rough sc_mul(Rough a, Rough b) { return {a.v * b.v}; }
Rough sc_neg(Rough a) { return {-a.v}; }
Rough sc_fma2(Rough a, Rough b) { return {2.0 * a.v + b.v}; }
Rough sc_fma_half(Rough a, Rough b) { return {0.5 * a.v + b.v}; }
Rough sc_near(Rough a) { return a; }

// the map's bound for states within lim
void bound_within(ScreenPlan& plan, const double* lim, MapBound& b)
{
  const Domain& dom = plan.dom;
  // the start points: a few roundings of |c| + r (1 + |g|) on either side, and of the shift
  double e0[B12G_MAX_DIM] = {0.0, 0.0, 0.0, 0.0};
  for (int j = 0; j < plan.dim; ++j) {
    const double shift = plan.kind == B12G_MAP_LORENZ && j == 2 ? std::fabs(plan.map.p[1]) : 0.0;
    e0[j] = 64.0 * kU * (std::fabs(dom.c[j]) + shift + 8.0 * dom.r[j] * (1.0 + plan.gmax));
  }
  if (plan.kind == B12G_MAP_LORENZ) lorenz_bound(plan.map, lim, e0, b, plan.k);
  else if (plan.kind == B12G_MAP_FORCED_DUFFING) forced_bound(plan.map, lim, e0, b, plan.k);
  else coupled_bound(plan.map, lim, e0, b, plan.k);
}

// How far from the shift the domain's trajectories go where the kernels look, from its
// corners and its centre: an estimate, nothing is proven from it.  Trajectories that leave 64
// times the domain are left out.
void estimate_reach(const ScreenPlan& plan, const double* base, const MapBound& b, double* reach)
{
  const int dim = plan.dim;
  const uint32_t steps = plan.map.steps;
  Rough k[kScreenCoef];
  for (int i = 0; i < kScreenCoef; ++i) k[i].v = plan.k[i];
  std::vector<double> force;
  if (plan.kind == B12G_MAP_FORCED_DUFFING) {
    force.resize(2 * size_t(steps) + 1);
    for (size_t i = 0; i < force.size(); ++i) force[i] = plan.k[3] * std::cos(0.5 * double(i) * plan.map.h);
  }
  const int corners = 1 << dim;
  for (int j = 0; j < dim; ++j) reach[j] = 0.0;
  for (int p = 0; p <= corners; ++p) {
    double most[B12G_MAX_DIM] = {}, at[B12G_MAX_DIM] = {};
    for (int j = 0; j < dim; ++j) {
      const double off = p == corners ? 0.0 : (p >> j) & 1 ? 1.0 : -1.0;
      at[j] = b.scale[j] * (plan.dom.c[j] + off * plan.dom.r[j] - b.shift[j]);
    }
    bool kept = true;
    auto look = [&](const Rough* x, int first, int end) {
      for (int j = first; j < end; ++j) {
        const double v = std::fabs(x[j].v / b.scale[j]);
        most[j] = std::max(most[j], v);
        kept = kept && v <= 64.0 * base[j];
      }
    };
    if (plan.kind == B12G_MAP_LORENZ) {
      Rough x[3] = {{at[0]}, {at[1]}, {at[2]}};
      for (uint32_t i = 0; i < steps && kept; ++i) {
        look(x, 0, 3);
        lorenz_screen_step(k, x);
      }
    } else if (plan.kind == B12G_MAP_FORCED_DUFFING) {
      Rough x[2] = {{at[0]}, {at[1]}};
      for (uint32_t i = 0; i < steps && kept; ++i) {
        look(x, 0, 2);
        forced_screen_step(k, Rough{force[2 * i]}, Rough{force[2 * i + 1]}, Rough{force[2 * i + 2]}, x);
      }
    } else {
      Rough x[4] = {{at[0]}, {at[1]}, {at[2]}, {at[3]}};
      look(x, 2, 4);
      duffing_screen_half_drift(x);
      for (uint32_t i = 0; i < steps && kept; ++i) {
        if (i) duffing_screen_drift(x);
        look(x, 0, 2);
        duffing_screen_kick(k, x);
      }
    }
    for (int j = 0; j < dim && kept; ++j) reach[j] = std::max(reach[j], most[j]);
  }
}

// the limits of candidate `tr`: the trajectories' estimated reach first, then multiples of
// the domain
void candidate_limits(ScreenPlan& plan, int tr, double* lim)
{
  static const double kLambda[kScreenBoxes] = {0.0, 2.0, 1.75, 1.5, 1.25, 1.1, 1.0};
  double base[B12G_MAX_DIM];
  for (int j = 0; j < plan.dim; ++j) {
    const double shift = plan.kind == B12G_MAP_LORENZ && j == 2 ? plan.map.p[1] : 0.0;
    base[j] = std::fabs(plan.dom.c[j] - shift) + plan.dom.r[j];
    // (the forced map's velocity enters the bound little, so its limit is twice as wide)
    if (plan.kind == B12G_MAP_FORCED_DUFFING && j == 1) base[j] *= 2.0;
    lim[j] = kLambda[tr] * base[j];
  }
  if (tr > 0) return;
  MapBound b;
  double reach[B12G_MAX_DIM];
  bound_within(plan, base, b);                // (its scales and the coefficients)
  estimate_reach(plan, base, b, reach);
  for (int j = 0; j < plan.dim; ++j) {
    lim[j] = std::max(base[j], 1.125 * reach[j]);
    plan.wide = plan.wide || lim[j] > 2.0 * base[j];
  }
}

}  // namespace

// The screened evaluation applies when the parameters are moderate, every dimension has at
// most kScreenMaxBits bisections and the share P of the points within the guard of a box
// boundary, if they lie evenly, is small.  The wider the limits, the fewer trajectories leave
// them and the larger E.  First come the limits that the domain's trajectories are estimated
// to need, where those go beyond twice the domain, then the widest of a few multiples of the
// domain that keeps P under 2^-12 (one warp in 128 evaluates again), else the domain itself
// if it keeps P under 2^-9 (one in 16).  Points whose trajectories leave the limits come on
// top: a warp with an undecided point runs both evaluations.
// The estimate is for domains that trajectories leave on their way and come back to, as
// around a saddle.  Images of 200,000 boxes: Lorenz (125 points), centre 0, radius 5, 1.25 ms
// against 2.87 with limits of twice the domain and 2.28 (strict) or 1.43 (FMA) in the map's
// own arithmetic; forced Duffing (16 points), radius 0.5, 1.15 ms against 3.43 and 2.45.
void screen_at(ScreenPlan& plan, int depth, ScreenArgs& s)
{
  s.on = 0;
  if (!plan.possible) return;
  const Domain& dom = plan.dom;
  const int dim = plan.dim;
  DepthConst dc;
  fill_depth_const(dom, dim, depth, dc);
  for (int j = 0; j < dim; ++j)
    if (dc.k[j] > kScreenMaxBits) return;
  for (int tr = 0; tr < kScreenBoxes; ++tr) {
    MapBound& b = plan.bound[tr];
    if (!plan.found[tr]) {
      double lim[B12G_MAX_DIM];
      candidate_limits(plan, tr, lim);
      bound_within(plan, lim, b);
      plan.found[tr] = true;
    }
    if (tr == 0 && !plan.wide) continue;
    double share = 0.0;
    bool ok = true;
    for (int j = 0; j < dim; ++j) {
      if (!(b.E[j] <= kEta * b.lim[j])) { ok = false; break; }
      // in boxes: the distance, the roundings of the exact index and of the domain's
      // faces, those of the screened position, and the fixed-point form's
      const double half = 0.5 * dc.ax[j].pk;
      const double g = half * (b.E[j] + 64.0 * kU * (std::fabs(dom.c[j]) + std::fabs(b.shift[j]) + 4.0 * dom.r[j])) /
                           dom.r[j] * (1.0 + 0x1p-20) + 0x1p-30;
      share += 2.0 * g;
      if (!(g < 0.125)) { ok = false; break; }
      s.guard[j] = uint32_t(std::ceil(g * 0x1p32)) + 2u;
    }
    if (!ok || !(share <= (tr == kScreenBoxes - 1 ? 0x1p-9 : 0x1p-12))) continue;
    for (int j = 0; j < dim; ++j) {
      const double S = b.scale[j], r = dom.r[j], rk = dc.ax[j].rk, half = 0.5 * dc.ax[j].pk;
      s.E[j] = b.E[j];
      s.sA[j] = 2.0 * r * S;
      s.sB[j] = S * ((dom.c[j] - b.shift[j]) - 3.0 * r + rk);
      s.sC[j] = S;
      s.sD[j] = -S * b.shift[j];
      s.sR[j] = S * rk;
      s.sP[j] = s.sD[j] - 3.0 * s.sR[j];
      s.tA[j] = half / (r * S);
      s.tB[j] = 0x1.8p20 + (half + half * (b.shift[j] - dom.c[j]) / r);
      s.bits[j] = uint32_t(dc.k[j]);
      // |X| < L is certain when the high word of |X| is below that of L
      const double L = std::fabs(S) * b.lim[j];
      unsigned long long w;
      __builtin_memcpy(&w, &L, sizeof w);
      const uint32_t hi = uint32_t(w >> 32) - 1u;
      __builtin_memcpy(&s.lim[j], &hi, sizeof hi);
    }
    for (int i = 0; i < kScreenCoef; ++i) s.k[i] = plan.k[i];
    s.on = 1;
    return;
  }
}

void fill_screen(uint32_t map_kind, const MapParams& map, const Domain& dom, int dim, int depth, double gmax,
                 ScreenPlan* plan, ScreenArgs& s)
{
  ScreenPlan here;
  if (!plan) plan = &here;
  const bool same = plan->dim == dim && plan->kind == map_kind && plan->map.steps == map.steps &&
                    std::memcmp(&plan->map.h, &map.h, sizeof map.h) == 0 &&
                    std::memcmp(plan->map.p, map.p, sizeof map.p) == 0 &&
                    std::memcmp(&plan->gmax, &gmax, sizeof gmax) == 0;
  if (!same) *plan = screen_plan(map_kind, map, dom, dim, gmax);
  screen_at(*plan, depth, s);
}

bool screen_record(uint32_t map_kind, int dim, const ScreenArgs& s, ScreenArgs& common, ScreenRec& rec)
{
  rec = ScreenRec{};
  if (!s.on) return true;
  // the coefficients an instance may have of its own (Screen<Map>::own)
  int own[2] = {-1, -1};
  if (map_kind == B12G_MAP_LORENZ) { own[0] = 5; own[1] = 9; }
  else if (map_kind == B12G_MAP_FORCED_DUFFING) own[0] = 3;
  else return false;
  if (!common.on) {
    common = s;
  } else {
    for (int i = 0; i < kScreenCoef; ++i)
      if (i != own[0] && i != own[1] && std::memcmp(&s.k[i], &common.k[i], sizeof(double)) != 0) return false;
    for (int j = 0; j < dim; ++j)
      if (std::memcmp(&s.sA[j], &common.sA[j], sizeof(double)) != 0) return false;
  }
  for (int i = 0; i < 2; ++i) rec.own[i] = own[i] >= 0 ? s.k[own[i]] : 0.0;
  for (int j = 0; j < dim; ++j) {
    rec.sB[j] = s.sB[j];
    rec.tB[j] = s.tB[j];
    rec.sR[j] = s.sR[j];
    rec.tA[j] = s.tA[j];
    rec.guard[j] = s.guard[j];
    rec.lim[j] = s.lim[j];
    rec.k |= s.bits[j] << (8 * j);
  }
  rec.on = 1;
  return true;
}

namespace {

uint32_t high_word(double x)
{
  unsigned long long w;
  std::memcpy(&w, &x, sizeof w);
  return uint32_t(w >> 32);
}

// one point on the host: the operations of the kernels' screened() and screen_locate()
bool host_kept(const ScreenArgs& s, int first, int end, const double* x)
{
  for (int j = first; j < end; ++j) {
    uint32_t lim;
    std::memcpy(&lim, &s.lim[j], sizeof lim);
    if ((high_word(x[j]) & 0x7FFFFFFFu) > lim) return false;
  }
  return true;
}

bool host_run(const ScreenArgs& s, uint32_t kind, const MapParams& map, double* x)
{
  bool kept = true;
  if (kind == B12G_MAP_LORENZ) {
    double y[3] = {x[0], x[1], x[2]};
    for (uint32_t i = 0; i < map.steps; ++i) {
      kept = kept && host_kept(s, 0, 3, y);
      lorenz_screen_step(s.k, y);
    }
    std::copy(y, y + 3, x);
  } else if (kind == B12G_MAP_FORCED_DUFFING) {
    double y[2] = {x[0], x[1]};
    const auto force = [&](uint32_t j) {      // the kernels read the cosines from a table made like this
      return s.k[3] * std::cos(double(j) * (map.h * double(map.steps) / double(2 * map.steps)));
    };
    for (uint32_t i = 0; i < map.steps; ++i) {
      kept = kept && host_kept(s, 0, 2, y);
      forced_screen_step(s.k, force(2 * i), force(2 * i + 1), force(2 * i + 2), y);
    }
    std::copy(y, y + 2, x);
  } else {
    double y[4] = {x[0], x[1], x[2], x[3]};
    kept = host_kept(s, 2, 4, y);
    duffing_screen_half_drift(y);
    for (uint32_t i = 0; i < map.steps; ++i) {
      if (i) duffing_screen_drift(y);
      kept = kept && host_kept(s, 0, 2, y);
      duffing_screen_kick(s.k, y);
    }
    duffing_screen_half_drift(y);
    std::copy(y, y + 4, x);
  }
  return kept;
}

}  // namespace

}  // namespace b12g

using namespace b12g;
using namespace b12g::host;

extern "C" b12g_status b12g_screen_probe(const b12g_domain* domain, const b12g_map* m, uint8_t depth, double reach,
                                         const uint64_t* codes, const double* offsets, uint64_t n, int from_centre,
                                         int* applies, double* bound, double* images, uint8_t* decided,
                                         uint64_t* boxes)
{
  if (!domain || !m || !applies || (n && (!codes || !offsets || !images || !decided || !boxes)))
    return fail(B12G_ERR_INVALID, "NULL argument");
  const int D = int(domain->dim);
  if (D < 1 || D > B12G_MAX_DIM || depth > 64 || !image_supported(m->kind, m->arith, B12G_GRID_PHILOX, domain->dim))
    return fail(B12G_ERR_INVALID, "unsupported map, dimension or depth");
  Domain dom;
  fill_domain(*domain, dom);
  MapParams mp;
  fill_map(*m, mp);
  ScreenArgs s{};
  fill_screen(m->kind, mp, dom, D, int(depth), reach, nullptr, s);
  *applies = s.on;
  if (!s.on) return B12G_OK;
  if (bound)
    for (int j = 0; j < D; ++j) bound[j] = s.E[j];
  for (uint64_t i = 0; i < n; ++i) {
    double x[B12G_MAX_DIM] = {};
    for (int j = 0; j < D; ++j) {
      uint32_t index = 0;
      for (int t = j; t < int(depth); t += D) index = (index << 1) | uint32_t((codes[i] >> (depth - 1 - t)) & 1u);
      const double v = 1.0 + double(index) * pow2_hd(-int(s.bits[j]));
      // (the centre in the order of box_axis)
      const double t = double(index) * pow2_hd(1 - int(s.bits[j])) - 1.0;
      const double centre = (t * dom.r[j] + dom.c[j]) + dom.r[j] * pow2_hd(-int(s.bits[j]));
      const double start = from_centre ? sc_fma(centre, s.sC[j], s.sD[j]) : sc_fma(v, s.sA[j], s.sB[j]);
      x[j] = sc_fma(offsets[i * D + j], s.sR[j], start);
    }
    bool sure = host_run(s, m->kind, mp, x), inside = true;
    uint32_t at[B12G_MAX_DIM] = {};
    for (int j = 0; j < D; ++j) {
      const double t = sc_fma(x[j], s.tA[j], s.tB[j]);
      unsigned long long w;
      std::memcpy(&w, &t, sizeof w);
      at[j] = uint32_t(w >> 32) - 0x41380000u;
      sure = sure && uint32_t(w) - s.guard[j] <= ~(2u * s.guard[j]);
      inside = inside && (at[j] >> s.bits[j]) == 0u;
      images[i * D + j] = (x[j] - s.sD[j]) / s.sC[j];
    }
    decided[i] = sure ? 1 : 0;
    uint64_t code = 0;
    for (int t = 0; t < int(depth); ++t) code = (code << 1) | ((at[t % D] >> (s.bits[t % D] - 1 - t / D)) & 1u);
    boxes[i] = inside ? code : kInvalidCode;
  }
  return B12G_OK;
}
