// The bound of the near / far split (rd_near.cuh, rd_tipnear.cuh) against the pair sums: after
// an emission every chain keeps the estimate of the field at its last point and the bound on
// it, and the last pass has formed the pair sum there.  Two diodes, so that the chains' state
// is in memory throughout.  Linked with the library; prints, per state, the chains compared
// and the largest |estimate - pair sum| / bound, and fails above 1.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "../rumdeed_gb300/csrc/rd_pair.cuh"
#include "rumdeed_gpu.h"

int rd_engine_chains(rd_engine* e, int diode, ChainState* cs, long long* first);

#define RD(x) do { if (int rc_ = (x)) { printf("%s: %d %s\n", #x, rc_, rd_last_error()); exit(2); } } while (0)

template <class T>
static std::vector<T> host(const T* p, long long first, int n) {
  std::vector<T> v(n);
  if (cudaMemcpy(v.data(), p + first, sizeof(T) * n, cudaMemcpyDeviceToHost) != cudaSuccess) exit(3);
  return v;
}

struct Case {
  const char* name;
  int tip, precision, n, max_chains;
  double side, low, high;   // emitter side; heights of the electrons, log-uniform (nm)
  bool at_nodes;            // beside the supply rule's nodes
};

static bool check(const Case& c) {
  std::mt19937_64 rng(c.n + 7 * c.precision);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  rd_diode_config d = {};
  d.geometry = c.tip ? RD_GEOM_TIP : RD_GEOM_PLANAR;
  d.V_s = c.tip ? 3000.0 : 2000.0;
  d.gap = 1.0e-6;
  d.time_step = 0.25e-15;
  d.image_charge = 1;
  d.capacity = c.n + 4000;
  d.max_chains = c.max_chains;
  d.emission = 1;
  d.mh_jumps = 40;
  const double phi = 2.0;
  d.work = &phi;
  d.work_nx = d.work_ny = 1;
  std::vector<double> pos;
  const double nm = 1.0e-9, pi = 3.14159265358979323846;
  if (c.tip) {
    const double h = 5.0e-7, dt = 1.0e-6, R = std::sqrt(250.0e-9 * (h * h / dt + 2.0 * h));
    d.tip_dim[0] = dt; d.tip_dim[1] = R; d.tip_dim[2] = h;
    d.tip_work_function = 2.5;
    const double a = std::sqrt(dt * dt * R * R / (h * h + 2.0 * dt * h) + dt * dt), eta1 = -dt / a, xm = h / dt + 1.0;
    for (int k = 0; k < c.n; ++k) {   // c.low of the way from the surface at least
      const double xi = 1.0 + 0.9 * (xm - 1.0) * u(rng), eta = eta1 * (1.0 - c.low * std::pow(c.high / c.low, u(rng))), ph = 2.0 * pi * u(rng);
      const double r = a * std::sqrt((xi * xi - 1.0) * (1.0 - eta * eta));
      pos.insert(pos.end(), {r * std::cos(ph), r * std::sin(ph), a * xi * eta + std::fabs(a * eta1 * xm)});
    }
  } else {
    const double L = c.side * nm;
    d.emitter_pos[0] = d.emitter_pos[1] = -0.5 * L;
    d.emitter_dim[0] = d.emitter_dim[1] = L;
    long long points = 0;
    RD(rd_supply_points(&d, &points));
    const int P = (int)std::lround(std::sqrt((double)points)) / 4;
    const double t[4] = {-0.86113631159405258, -0.33998104358485626, 0.33998104358485626, 0.86113631159405258};
    for (int k = 0; k < c.n; ++k) {
      const double z = c.low * std::pow(c.high / c.low, u(rng)), ang = 2.0 * pi * u(rng);
      double x = (u(rng) - 0.5) * c.side, y = (u(rng) - 0.5) * c.side;
      if (c.at_nodes) {   // z / 2 off a node: where its field changes fastest
        x = (-0.5 + ((int)(P * u(rng)) + 0.5 * (1.0 + t[(int)(4 * u(rng))])) / P) * c.side + 0.5 * z * std::cos(ang);
        y = (-0.5 + ((int)(P * u(rng)) + 0.5 * (1.0 + t[(int)(4 * u(rng))])) / P) * c.side + 0.5 * z * std::sin(ang);
      }
      pos.insert(pos.end(), {x * nm, y * nm, z * nm});
    }
  }
  long long points = 0;
  RD(rd_supply_points(&d, &points));
  rd_engine_config ec = {};
  ec.precision = c.precision;
  ec.max_diodes = 2;
  ec.particle_capacity = 2LL * (d.capacity + 64);
  ec.chain_capacity = 2LL * (c.max_chains + 64);
  ec.quad_capacity = 2 * points + 128;
  rd_engine* e = nullptr;
  RD(rd_engine_create(&ec, &e));
  double worst = 0.0;
  long long compared = 0;
  int id[2];
  for (int k = 0; k < 2; ++k) {
    d.seed = 11 + k;
    RD(rd_diode_add(e, &d, &id[k]));
    RD(rd_add_particles(e, id[k], c.n, pos.data(), nullptr, nullptr, 0, 1));
  }
  for (int step = 1; step <= 2; ++step) {
    RD(rd_do_emission(e, step));
    for (int k = 0; k < 2; ++k) {
      rd_counters y;
      RD(rd_counters_get(e, id[k], &y));
      ChainState cs;
      long long first = 0;
      RD(rd_engine_chains(e, id[k], &cs, &first));
      const std::vector<float> est = host(cs.fF, first, y.chains), bound = host(cs.fe, first, y.chains);
      const std::vector<double> F = host(cs.F, first, y.chains);
      const std::vector<int> ok = host(cs.ok, first, y.chains);
      for (int q = 0; q < y.chains; ++q)
        if (ok[q] && bound[q] > 0.0f) {
          const double r = std::fabs((double)est[q] - F[q]) / bound[q];
          worst = r > worst || std::isnan(r) ? r : worst;
          ++compared;
        }
    }
  }
  RD(rd_engine_destroy(e));
  printf("%-28s %7lld chains, largest |estimate - pair sum| / bound %.3f\n", c.name, compared, worst);
  return compared > 100 && worst <= 1.0;
}

int main() {
  const Case cases[] = {
      {"fp32 layer", 0, RD_PREC_FP32C, 4000, 20000, 1000.0, 0.5, 400.0, false},
      {"fp32 nodes 20 um", 0, RD_PREC_FP32C, 20000, 20000, 20000.0, 0.05, 1.5, true},
      {"fp32 small, many near", 0, RD_PREC_FP32C, 8000, 8000, 300.0, 3.0, 60.0, false},
      {"fp64 layer", 0, RD_PREC_FP64, 2000, 8000, 1000.0, 0.5, 400.0, false},
      {"fp64 nodes 2 um", 0, RD_PREC_FP64, 5000, 8000, 2000.0, 0.05, 1.5, true},
      {"fp64 nodes 8 um", 0, RD_PREC_FP64, 20000, 8000, 8000.0, 0.05, 1.5, true},
      {"fp64 nodes 20 um", 0, RD_PREC_FP64, 20000, 8000, 20000.0, 0.05, 1.5, true},
      {"fp64 nodes 20 um, 1 nm", 0, RD_PREC_FP64, 20000, 8000, 20000.0, 0.9, 1.3, true},
      {"fp64 touching", 0, RD_PREC_FP64, 60, 2000, 300.0, 1.0e-6, 1.0e-2, true},
      {"tip close", 1, RD_PREC_FP32C, 4000, 8000, 0.0, 0.002, 0.1, false},
      {"tip spread", 1, RD_PREC_FP32C, 8000, 8000, 0.0, 0.05, 0.9, false},
  };
  bool good = true;
  for (const Case& c : cases) good = check(c) && good;
  return good ? 0 : 1;
}
