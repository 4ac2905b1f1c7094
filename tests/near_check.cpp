// Host check of rd_bounds.h: the sums of the planar near / far split, added in the order
// and the arithmetic of rd_near.cuh's kernels, against the same sums in double.  The
// terms are chosen so that the roundings agree: one large term, then runs that lie just
// below half an ulp of the sum so far and are lost one by one.  A bound's share for such
// a sum is what it leaves beside the pair sum's 153 u, a term's 25 u and the evaluation's
// 30 u.  Prints the worst error over its share.
#include <cmath>
#include <cstdio>
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

int main() {
  for (int cnt : {0, 1, 8, 255, 256, 257, 1024, 4096, 6000, 20000, 100000, 1000000}) {
    for (int P : {16, 256, 1024}) {
      // the points' own coordinates are another matter: without the 0.6 P
      check(0, 8, RD_NEAR_RUN, cnt, rd_near_units(P, cnt) - 0.6f * P, 1.0);
      check(1, 2, RD_NEAR_RUN, cnt, RD_NEAR_UNITS * rd_near_node_factor(cnt), 1.0);
    }
    for (int nt : {128, 256}) check(2, nt, 8, cnt, rd_near_direct_units(cnt, nt), 1.0);
  }
  printf("point %.3f node %.3f direct %.3f\n", worst[0], worst[1], worst[2]);
  return !(worst[0] <= 1.0 && worst[1] <= 1.0 && worst[2] <= 1.0);
}
