// The jumps' counters that a step left half full (a wait that gave up) are zero again before
// the next step's first jump: the set-up launches of rd_near.cuh and rd_tipnear.cuh on one
// diode each, with one electron and no item of work, so that every index is 0 or within the
// arrays below.  Linked with the library; prints the counters and progress words.
#include <cstdio>
#include <vector>
#include "../rumdeed_gb300/csrc/rd_pair.cuh"

cudaError_t rd_launch_near_setup(int prec, int nslots, int grid, cudaStream_t st, const DiodeParams* P, const DiodeDyn* Dy,
                                 const Pool& pool, const PlanEntry* sup_plan, const PlanHeader* sup_ph,
                                 const float4* qpp, const double* qF, const NearState& nr, double kscale);
cudaError_t rd_launch_tip_near(int nslots, int grid, cudaStream_t st, const DiodeParams* P, DiodeDyn* Dy,
                               const Pool& pool, const PlanEntry* plan, const PlanHeader* ph, const PlanEntry* plan_mh,
                               const ChainState& cs, const int* ch_off, const int* step_ptr, int jumps,
                               const NearState& nr, double kscale, int* gave_up);

template <class T>
static T* device(size_t n, int byte = 0) {
  T* p = nullptr;
  if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess || cudaMemset(p, byte, n * sizeof(T)) != cudaSuccess) return nullptr;
  return p;
}

int main() {
  DiodeParams p{};
  p.active = p.emission = p.mh_fast = p.image_charge = 1;
  p.geometry = RD_G_PLANAR;
  p.cap = 32;
  p.nr_P = 16; p.nr_bx = 22; p.nr_by = 11;
  p.nr_iwx = p.nr_iwy = 1.0f; p.nr_Z = 1.0f;
  p.mh_hi = 0.125;
  DiodeDyn y{};
  y.n = 1; y.chains = 5; y.MH_std = 0.0625;
  DiodeParams* P = device<DiodeParams>(1);
  DiodeDyn* Dy = device<DiodeDyn>(1);
  PlanEntry* plan = device<PlanEntry>(1);
  PlanHeader* ph = device<PlanHeader>(1);   // no items
  Pool pool{};
  pool.zk_hi = device<float4>(32); pool.zk_lo = device<float4>(32);
  pool.pk_hi = device<float4>(32); pool.pk_lo = device<float4>(32);
  NearState nr{};
  nr.low = device<float4>(32); nr.hi = device<float4>(32); nr.lo = device<float2>(32);
  nr.rank = device<int>(32); nr.cnt = device<int>(1024); nr.start = device<int>(1024); nr.rec = device<float>(1024);
  nr.count = device<unsigned long long>(4, 0x11); nr.progress = device<unsigned long long>(4, 0x11);
  nr.ring = device<unsigned long long>(16, 0x11);
  int* ints = device<int>(64);
  double* qF = device<double>(64);
  float4* qpp = device<float4>(64);
  int bad = 0;
  for (int tip = 0; tip < 2; ++tip) {
    if (tip) { p.geometry = RD_G_TIP; p.mh_fast = 0; p.tn = 1; p.tn_np = 0; p.h_tip = 2.0e-7; p.r_tip = 1.0e-7; }
    cudaMemset(nr.count, 0x11, 4 * sizeof(unsigned long long));
    cudaMemcpy(P, &p, sizeof p, cudaMemcpyHostToDevice);
    cudaMemcpy(Dy, &y, sizeof y, cudaMemcpyHostToDevice);
    cudaError_t e = tip ? rd_launch_tip_near(1, 1, nullptr, P, Dy, pool, plan, ph, plan, ChainState{}, ints, ints, 1, nr, 1.0, ints)
                        : rd_launch_near_setup(1, 1, 1, nullptr, P, Dy, pool, plan, ph, qpp, qF, nr, 1.0);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    unsigned long long count = 1, progress = 0;
    cudaMemcpy(&count, nr.count, sizeof count, cudaMemcpyDeviceToHost);
    cudaMemcpy(&progress, nr.progress, sizeof progress, cudaMemcpyDeviceToHost);
    printf("%s: error %d count %llx progress %llx\n", tip ? "tip" : "planar", (int)e, count, progress);
    bad |= e != cudaSuccess || count != 0 || (unsigned)progress != 0;
  }
  return bad;
}
