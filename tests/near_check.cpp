// Host check of rd_bounds.h: the sums of the planar near / far split, added in the order
// and the arithmetic of rd_near.cuh's kernels, against the same sums in double.  The
// terms are chosen so that the roundings agree: one large term, then runs that lie just
// below half an ulp of the sum so far and are lost one by one.  A bound's share for such
// a sum is what it leaves beside the pair sum's 153 u, a term's 25 u and the evaluation's
// 30 u.  And the guard of a decision: df and log u in FP32, each logarithm moved by an ulp
// either way, against FP64, for planar and tip targets.  Prints the worst error over its
// share.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "../rumdeed_gb300/csrc/rd_bounds.h"

static double worst[3];
static void note(int k, double err, double mag, double units) {
  const double share = (units - (153.0 + 25.0 + 30.0)) * RD_U24 * mag;
  if (err > 0.0) worst[k] = std::fmax(worst[k], share > 0.0 ? err / share : INFINITY);
}

// One lane's share of a list: runs of `run` terms, each run then added to the sum.
static float lane_sum(const std::vector<float>& t, int run) {
  float s = 0.0f, r = 0.0f;
  for (size_t k = 0; k < t.size(); ++k) {
    r += t[k];
    if ((int)((k + 1) % run) == 0 || k + 1 == t.size()) { s += r; r = 0.0f; }
  }
  return s;
}

// n terms per lane whose runs round against the sum: the first is 1, the others add up to
// `part` of half an ulp per run.
static std::vector<float> terms(int n, int run, double part) {
  std::vector<float> t(n, (float)(part * 0x1p-24 / run));
  if (n > 0) t[0] = 1.0f;
  for (int k = 1; k < run && k < n; ++k) t[k] = 0.0f;
  return t;
}

static void check(int k, int lanes, int run, int cnt, double units, double scale) {
  for (double part : {0.5, 0.9, 0.99, 1.01, 1.5}) {
    const std::vector<float> t = terms((cnt + lanes - 1) / lanes, run, part);
    std::vector<float> s(lanes, lane_sum(t, run));
    double exact = 0.0;
    for (float v : t) exact += v;
    exact *= lanes;
    for (int w = lanes / 2; w > 0; w /= 2)
      for (int l = 0; l < w; ++l) s[l] += s[l + w];
    note(k, std::fabs((double)s[0] - exact) * scale, exact * scale, units);
  }
}

// The targets' difference less log u as near_decide forms them, from the fields Fn and Fc:
// `move` has a bit for each logarithm's direction.
struct Target {
  double logphi, lcoef, v;   // log phi, l_const / phi^2, xi^2 - eta^2 (planar: 1)
  bool tip;
};
static float ulp(float x, unsigned move, int bit) { return std::nextafterf(x, (move >> bit & 1) ? INFINITY : -INFINITY); }
static float rho_f(const Target& t, float F, unsigned move, int bit) {
  const float lphi = (float)t.logphi;
  float t0 = lphi, kf;
  if (t.tip) {
    const float m = rd_log_parts((float)t.v, &kf);
    t0 = rd_less_half_log(lphi, kf, ulp(std::log(m), move, bit));
  }
  const float l = (float)t.lcoef * (-F);
  float tau = 0.0f;
  if (l > 1.0f) tau = 1.0f / 9.0f;
  else if (l > 1.0e-30f) tau = l * ((1.0f / 9.0f) - (1.0f / 18.0f) * ulp(std::log(l), move, bit + 1));
  return std::fma(2.0f, ulp(std::log1p(tau), move, bit + 2), t0);
}
static double rho_d(const Target& t, double F) {
  const double l = std::fmin(t.lcoef * -F, 1.0), tau = l * (1.0 / 9.0 - std::log(l) / 18.0);
  return t.logphi - (t.tip ? 0.5 * std::log(t.v) : 0.0) + 2.0 * std::log1p(tau);
}

static double worst_guard;
static void check_guard() {
  std::mt19937_64 rng(5);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  for (int k = 0; k < 60000; ++k) {
    const bool tip = k & 1;
    Target n, c;
    n.tip = c.tip = tip;
    n.logphi = std::log(1.5 + 6.4 * u(rng));
    const double phi = std::exp(n.logphi), e2 = std::pow(10.0, -3.0 * u(rng));   // 1 - eta^2
    n.lcoef = 1.4e-9 / (phi * phi);
    c = n;
    const double top = std::pow(10.0, 2.0 * u(rng));
    n.v = tip ? std::pow(1.0 + top * u(rng), 2.0) - (1.0 - e2) : 1.0;
    c.v = tip ? std::pow(1.0 + top * u(rng), 2.0) - (1.0 - e2) : 1.0;
    if (tip && k % 5 == 0) {   // parts of rho that cancel
      n.v = phi * phi * (1.0 + 0.2 * u(rng));
      c.v = phi * phi * (1.0 + 0.2 * u(rng));
    }
    const double Fn = -std::pow(10.0, 7.0 + 3.5 * u(rng)), Fc = Fn * std::exp((u(rng) - 0.5) * (k % 3 ? 0.1 : 3.0));
    const double uu = k % 4 ? 1.0 - 1.0e-3 * u(rng) : u(rng);
    const float Fnf = (float)Fn, Fcf = (float)Fc, uf = (float)uu;
    const double d = 2.0 * std::log(Fn / Fc) - (rho_d(n, Fn) - rho_d(c, Fc));
    for (unsigned move = 0; move < 256; ++move) {
      const float l2 = 2.0f * ulp(std::log(Fnf / Fcf), move, 0), rn = rho_f(n, Fnf, move, 1), rc = rho_f(c, Fcf, move, 4);
      const float df = l2 - (rn - rc), lu = ulp(std::log(uf), move, 7);
      const float S = std::fabs(l2) + std::fabs(rn) + std::fabs(rc) + std::fabs(lu);
      worst_guard = std::fmax(worst_guard, std::fabs(((double)df - d) - ((double)lu - std::log(uu))) / rd_near_guard(S));
    }
  }
}

int main() {
  for (int cnt : {0, 1, 8, 255, 256, 257, 1024, 4096, 6000, 20000, 100000, 1000000}) {
    for (int P : {16, 256, 1024}) {
      // the points' own coordinates are another matter: without the 0.6 P
      check(0, 8, RD_NEAR_RUN, cnt, rd_near_units(P, cnt) - 0.6f * P, 1.0);
      check(1, 2, RD_NEAR_RUN, cnt, RD_NEAR_UNITS * rd_near_node_factor(cnt), 1.0);
    }
    for (int nt : {128, 256}) check(2, nt, 8, cnt, rd_near_direct_units(cnt, nt), 1.0);
  }
  check_guard();
  printf("point %.3f node %.3f direct %.3f guard %.3f\n", worst[0], worst[1], worst[2], worst_guard);
  return !(worst[0] <= 1.0 && worst[1] <= 1.0 && worst[2] <= 1.0 && worst_guard <= 1.0);
}
