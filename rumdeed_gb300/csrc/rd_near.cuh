// rd_near.cuh -- the jumps of the planar Metropolis-Hastings chains from a near /
// far split of the cathode field (included by rd_field.cu, in its anonymous
// namespace).
//
// A jump needs the field at its proposal only to compare two targets, and the
// FP32 chains already decide from FP32 estimates of the targets wherever those
// are certain (mh_decide_f).  (The FP64 form's chains take the same estimates, with
// FP64 points, draws and pair sums; below u and the pair sum's roundings are the FP32
// form's, the FP64 form's are smaller, but for what near_wide adds.)  The same holds for the field itself: an estimate
// with a bound on how far it can lie from the value the pair-sum kernel
// (k_mh_jump_planar) computes decides every jump outside that bound, and the few
// jumps inside it take sums over all electrons: first in any order, with a bound of
// their own, then as the pair-sum kernel forms them.  So the decisions, and with them
// the chains, are those of the pair-sum kernel, bit for bit, and the field that
// emission reads is the pair sum at the last point of each chain that has moved (one
// pass after the last jump, RD_MH_FINAL) and the start's field of the others.
//
// The estimate.  The step's supply integral has just evaluated the pair sum S at
// 4 x 4 Gauss-Legendre nodes of each of the emitter's P x P panels.  Electrons
// lower than nr_Z and within RD_NEAR_M panels of a panel (in whole bins) are near it; the others
// are far, and their part of S is smooth over the panel:
//   S(p) = I[S(nodes) - sum_near g(nodes)](p) + sum_near g(p),
// I the interpolation in the nodes, g_j(p) = q z / (rho^2 + z^2)^{3/2}.  A jump
// then costs 16 coefficients and the near electrons (tens to a few hundred)
// instead of all of them.
//
// The bound.  With a the panel's half widths and D the distance from a far
// electron to the panel, the Taylor coefficients of g along an axis are
// Gegenbauer polynomials of its direction cosine c, d^4 g / 4! = C_4^{3/2}(c) z / R^7,
// at most K z / D^7 with K = 15 (c = 1), or 2.5 where c^2 <= 0.68, so
//   |I g - g|(t) <= T_x |w(t_x)| a_x^4 + T_y L(t_x) |w(t_y)| a_y^4,
//   T = sum_far K z / D^7,  w(t) = prod (t - node),  L the Lebesgue function.
// The rounding of the pair sum itself (tiles of 128 terms added one after
// another: 128 u of the tile's sum of magnitudes, 25 u of each term), of the
// node values carried through I (L(t_x) L(t_y) times theirs), and of this
// kernel's own sums is bounded by multiples of u = 2^-24 times the sum of
// magnitudes, which is |S| because every charge has one sign (diodes that hold
// ions or atoms keep the pair-sum kernel).  near_bound0 and rd_bounds.h have the multiples.
//
// Measured (GB300, jumps of one step, the split's set-up and last pass included):
//   one diode, 4500 electrons, 3800 chains, 100 jumps      6.13 -> 0.67 ms
//   24 diodes of 256-4096 electrons, 30,000 chains, 200    15.9 -> 1.9 ms
//   128 diodes of 256-32768 electrons, 353,000 chains, 200  276 -> 22.3 ms
//   FP64: 1300 electrons, 960 chains, 100                   8.4 -> 0.85 ms
// Open after the estimate: one jump in 10^5; the estimate lies within 0.13 (FP32) and
// 0.30 (FP64) of its bound at the chains' last points (tests/near_bound.cu).  What is
// left is latency (one near list, one far record, three logarithms and one counter per
// jump), not arithmetic.
//
// Near region: RD_NEAR_M = 3 panels and nr_Z = 5 half widths.  5 panels and 8 half
// widths make the bound's T ten times smaller and leave half as many jumps open,
// but the near list more than twice as long: 31 -> 42 ms on the 128 diodes.

// Does the diode's step run its jumps here?  (planner mode PM_MH_NEAR)
__device__ __forceinline__ bool near_live(const DiodeParams& p, const DiodeDyn& y) {
  return p.active && p.emission && p.mh_fast && y.chains > 0 && !rd_mh_vacuum(p, y);
}

// Bin of a low electron: row << 16 | column, or -1 for one that is far from every
// panel.  Bins are one panel wide and two high, RD_NEAR_M panels more than the
// emitter on every side; the near region of panel (x, y) is the columns x .. x + 2 M
// and the RD_NEAR_ROWS rows from y / 2 on.
__device__ __forceinline__ int near_bin(const DiodeParams& p, float x, float y, float z) {
  if (!(z < p.nr_Z)) return -1;
  const float fx = floorf((x + p.em_hx) * p.nr_iwx), fy = floorf((y + p.em_hy) * p.nr_iwy);
  if (!(fabsf(fx) < 4096.0f) || !(fabsf(fy) < 4096.0f)) return -1;
  const int bx = (int)fx + RD_NEAR_M, y2 = (int)fy + RD_NEAR_M;
  if (bx < 0 || bx >= p.nr_bx || y2 < 0 || y2 >= 2 * p.nr_by) return -1;
  return ((y2 >> 1) << 16) | bx;
}

// A diode's progress through its jumps, written by the last tile of each jump: the
// number done, whether the step size is at its upper clamp (bit 31), and the step
// size as a float (high word).
#define RD_NEAR_CLAMPED 0x80000000u
__device__ __forceinline__ unsigned long long near_progress(const DiodeParams& p, int done, double mh_std) {
  return ((unsigned long long)__float_as_uint((float)mh_std) << 32) |
         ((unsigned)done | (mh_std == p.mh_hi ? RD_NEAR_CLAMPED : 0u));
}

// Before the first jump of a step: none done and none counted, also if a wait of the last
// step gave up half way through a jump.
__device__ __forceinline__ void near_reset(const DiodeParams& p, const NearState& nr, int d, double mh_std) {
  nr.progress[d] = near_progress(p, 0, mh_std);
  nr.count[d] = 0;
}

// Electrons into bins: each electron's bin and its rank among the bin's.
__global__ void __launch_bounds__(256)
k_near_count(const DiodeParams* __restrict__ P, const DiodeDyn* __restrict__ Dy, Pool pool, NearState nr) {
  const int d = blockIdx.y;
  const DiodeParams& p = P[d];
  if (!near_live(p, Dy[d])) return;
  const int n = Dy[d].n, nb = p.nr_bx;
  int* cnt = nr.cnt + p.nr_boff;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const float4 h = pool.zk_hi[p.off + j];
    const float z = pool.zk_lo[p.off + j].z;
    const int code = near_bin(p, h.x, h.y, z);
    nr.low[p.off + j] = make_float4(h.x, h.y, z, __int_as_float(code));
    if (code >= 0) nr.rank[p.off + j] = atomicAdd(&cnt[(code >> 16) * nb + (code & 0xffff)], 1);
  }
}

// First slot of each bin (one block per diode); the counts are left at zero for
// the next step.
__global__ void __launch_bounds__(1024)
k_near_scan(const DiodeParams* __restrict__ P, const DiodeDyn* __restrict__ Dy, NearState nr) {
  __shared__ int wsum[32];
  const int d = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const DiodeParams& p = P[d];
  if (!near_live(p, Dy[d])) return;
  const int bins = p.nr_bx * p.nr_by, per = (bins + 1023) / 1024;
  int* cnt = nr.cnt + p.nr_boff;
  int* start = nr.start + p.nr_boff;
  const int b0 = min(tid * per, bins), b1 = min(b0 + per, bins);
  int s = 0;
  for (int b = b0; b < b1; ++b) s += cnt[b];
  int x = s;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += v;
  }
  if (lane == 31) wsum[w] = x;
  __syncthreads();
  if (w == 0) {
    int t = wsum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += v;
    }
    wsum[lane] = t;
  }
  __syncthreads();
  int at = (w > 0 ? wsum[w - 1] : 0) + x - s;
  for (int b = b0; b < b1; ++b) {
    const int c = cnt[b];
    start[b] = at;
    cnt[b] = 0;
    at += c;
  }
  if (tid == 1023) start[bins] = at;   // the last thread's range ends at the last bin
  if (tid == 0) near_reset(p, nr, d, Dy[d].MH_std);
  if (tid < 4) nr.ring[4 * d + tid] = 0;
}

// The near electrons in bin order: (x_hi, y_hi, z^2, q z) and (x_lo, y_lo).
__global__ void __launch_bounds__(256)
k_near_scatter(const DiodeParams* __restrict__ P, const DiodeDyn* __restrict__ Dy, Pool pool, NearState nr) {
  const int d = blockIdx.y;
  const DiodeParams& p = P[d];
  if (!near_live(p, Dy[d])) return;
  const int n = Dy[d].n, nb = p.nr_bx;
  const int* start = nr.start + p.nr_boff;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const int code = __float_as_int(nr.low[p.off + j].w);
    if (code < 0) continue;
    const int k = p.off + start[(code >> 16) * nb + (code & 0xffff)] + nr.rank[p.off + j];
    const float4 l = pool.zk_lo[p.off + j];
    nr.hi[k] = pool.zk_hi[p.off + j];
    nr.lo[k] = make_float2(l.x, l.y);
  }
}

// The term of one electron at a point on the FP32 grid, or (qx, qy) off it.
__device__ __forceinline__ float near_term(float4 h, float2 l, float px, float py, float qx = 0.0f, float qy = 0.0f) {
  const float dx = (px - h.x) - (l.x - qx), dy = (py - h.y) - (l.y - qy);
  const float inv = rsqrtf(fmaf(dx, dx, fmaf(dy, dy, h.z)));
  return h.w * ((inv * inv) * inv);
}

// FP64 chains: how far a term can lie from the FP64 pair sum's, added to *wide.  The
// reference's r + l^2 (l^2 = 1e-9 nm) makes a term smaller by at most 3 l^2 / r of it.
// The packs and the split point hold a coordinate to 2^-48 of it and their difference
// loses as much again: 2^-45 of the emitter's half width together, which is at most
// 4 times that over r of the term as long as r is ten times larger; closer (and where
// l^2 shows in the first digit) nothing is promised.  At r = 1 nm this is 0.05 u of the
// term, at 1e-3 nm 50 u.
__device__ __forceinline__ float near_wide(const DiodeParams& p) {
  return 3.0e-9f + 1.2e-13f * (float)p.nr_P * fmaxf(p.nr_ax, p.nr_ay);
}
__device__ __forceinline__ float near_term(float4 h, float2 l, float px, float py, float qx, float qy, float kw,
                                           float* wide) {
  const float dx = (px - h.x) - (l.x - qx), dy = (py - h.y) - (l.y - qy);
  const float inv = rsqrtf(fmaf(dx, dx, fmaf(dy, dy, h.z))), g = h.w * ((inv * inv) * inv), k = kw * inv;
  *wide = fmaf(fabsf(g), k < 0.25f ? k : INFINITY, *wide);
  return g;
}

// Inverse Vandermonde matrix of the four Gauss-Legendre nodes: coefficients of
// the interpolating cubic from the node values.
__device__ const float c_gl4_inv[4][4] = {
    {-0.0923265988f, 0.592326599f, 0.592326599f, -0.0923265988f},
    {0.107214846f, -1.74223419f, 1.74223419f, -0.107214846f},
    {0.798762056f, -0.798762056f, -0.798762056f, 0.798762056f},
    {-0.927567512f, 2.34943118f, -2.34943118f, 0.927567512f}};

#define RD_NEAR_AWAY 24.0f    // electrons this many half widths from eight panels share their term of T

// Panel records, one warp per panel: the far part's interpolation coefficients
// (powers of t_x fastest), the panel's centre, T and the largest |S| of its
// nodes, and where its near electrons are.  A block takes the eight panels of a tile of
// the supply plan (128 points; the items of its first chunk).  T of every electron and
// panel, about 50 instructions a pair, was most of the set-up (128 diodes of 256-32768
// electrons, 230,000 panels: 11.2 ms, half of it on a part of the SMs only): electrons
// RD_NEAR_AWAY half widths from the eight panels' rectangle now add one term for all of
// them (at the rectangle's distance T is larger by a per cent or so), the others pass
// through shared memory once for the eight warps: 2.8 ms.
// S is the FP32 pair sum at the nodes' high words, or the FP64 one at the nodes
// themselves (high and low words); the near terms taken off it are at the same points:
// beside a node half an ulp of its coordinate is worth many of the bound's u.
template <int PREC>
__global__ void __launch_bounds__(256)
k_near_panels(const DiodeParams* __restrict__ P, const DiodeDyn* __restrict__ Dy, const PlanEntry* __restrict__ plan,
              const PlanHeader* __restrict__ ph, const float4* __restrict__ qpp, const double* __restrict__ qF,
              NearState nr, double kscale) {
  __shared__ float4 low[512];
  __shared__ float s_gT[8];
  __shared__ int s_n;
  const int total = ph->total_items, nd = ph->n_diodes, tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) s_n = 0;
  __syncthreads();
  const double inv_A0 = 1.0 / (-2.0 * kscale);
  for (int g = blockIdx.x; g < total; g += gridDim.x) {
    const ItemRef it = decode_item(plan, nd, g);
    const DiodeParams& p = P[it.d];
    if (it.chunk != 0 || !near_live(p, Dy[it.d])) continue;
    const int NP = p.nr_P, own = it.tile * 8 + (tid >> 5);
    const bool live = own < NP * NP;
    const int pan = live ? own : 0;   // (a warp without a panel helps to load)
    const int ppy = pan / NP, ppx = pan - ppy * NP, nb = p.nr_bx, r0 = ppy >> 1;
    const int* start = nr.start + p.nr_boff;
    // the node of this lane (lanes l and l + 16 share one and take every other near electron)
    const int k = p.q_off + (ppy * 4 + ((lane >> 2) & 3)) * p.quad_n + ppx * 4 + (lane & 3);
    const float4 pp = qpp[k];
    const float S = (float)((qF[k] - p.E_z) * inv_A0);
    float near = 0.0f, wide = 0.0f;
    const float kw = near_wide(p);
    int cnt = 0;   // near electrons
    for (int r = 0; r < RD_NEAR_ROWS; ++r) {
      const int row = (r0 + r) * nb + ppx;   // bins ppx .. ppx + 2 M of this row
      const int e1 = start[row + RD_NEAR_W];
      cnt += e1 - start[row];
      for (int e0 = start[row]; e0 < e1; e0 += 64) {   // short runs: the sums stay accurate
        float s = 0.0f;
        for (int e = e0 + (lane >> 4); e < min(e0 + 64, e1); e += 2)
          s += PREC == 1 ? near_term(nr.hi[p.off + e], nr.lo[p.off + e], pp.x, pp.z)
                         : near_term(nr.hi[p.off + e], nr.lo[p.off + e], pp.x, pp.z, pp.y, pp.w, kw, &wide);
        near += s;
      }
    }
    near += __shfl_xor_sync(0xffffffffu, near, 16);
    float big = fabsf(S);
    if (PREC == 0) {   // the node's near terms too, in the units of the bound on `big`'s
      wide += __shfl_xor_sync(0xffffffffu, wide, 16);
      big = fmaf(wide, 1.0f / (RD_U24 * RD_NEAR_UNITS), big);
      if (!(big < INFINITY)) big = INFINITY;
    }
    for (int o = 8; o > 0; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
    big *= rd_near_node_factor(cnt);
    // tensor coefficients of the far part, about the value at the first node
    const float far = S - near, base = __shfl_sync(0xffffffffu, far, 0), v = far - base;
    float cx = 0.0f, c = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) cx = fmaf(c_gl4_inv[lane & 3][q], __shfl_sync(0xffffffffu, v, (lane & 12) + q), cx);
#pragma unroll
    for (int q = 0; q < 4; ++q) c = fmaf(c_gl4_inv[(lane >> 2) & 3][q], __shfl_sync(0xffffffffu, cx, 4 * q + (lane & 3)), c);
    if (lane == 0) c += base;
    // T over the far electrons, as seen from the panel's rectangle
    const float ox = (float)((2 * ppx + 1 - NP) * p.nr_hx), oy = (float)((2 * ppy + 1 - NP) * p.nr_hy);
    const float ax = p.nr_ax, ay = p.nr_ay;
    float Tx = 0.0f, Ty = 0.0f, gT = 0.0f;
    const int n = Dy[it.d].n;
    // electrons far from all eight panels (a row of them, or parts of two): one term for
    // all, at the least distance to their rectangle; the others go to every warp
    const int g0 = it.tile * 8, g1 = min(g0 + 7, NP * NP - 1), ra = g0 / NP, rb = g1 / NP;
    const int ca = ra == rb ? g0 - ra * NP : 0, cb = ra == rb ? g1 - rb * NP : NP - 1;
    const float gx = (float)((ca + cb + 1 - NP) * p.nr_hx), gy = (float)((ra + rb + 1 - NP) * p.nr_hy);
    const float hx = (float)(cb - ca + 1) * ax * 1.0001f, hy = (float)(rb - ra + 1) * ay * 1.0001f;
    const float away = RD_NEAR_AWAY * fmaxf(ax, ay), away2 = away * away;
    int here = 0;   // electrons in low
    for (int j0 = 0; j0 < n; j0 += 256) {
      float4 e4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      bool close = false;
      if (j0 + tid < n) {
        e4 = nr.low[p.off + j0 + tid];
        const float bx = fmaxf(fabsf(e4.x - gx) - hx, 0.0f), by = fmaxf(fabsf(e4.y - gy) - hy, 0.0f);
        const float r2 = fmaf(bx, bx, fmaf(by, by, e4.z * e4.z));
        close = r2 < away2;
        if (!close) {
          const float inv = rsqrtf(r2), i2 = inv * inv;
          gT = fmaf(e4.z * inv, i2 * i2 * i2, gT);
        }
      }
      const unsigned mask = __ballot_sync(0xffffffffu, close);
      int at = 0;
      if (lane == 0 && mask) at = atomicAdd(&s_n, __popc(mask));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (close) low[at + __popc(mask & ((1u << lane) - 1))] = e4;
      here += __syncthreads_count(close);
      if (here <= 256 && j0 + 256 < n) continue;   // room for another 256 (block-uniform)
#pragma unroll 4
      for (int q = lane; q < here; q += 32) {
        const float4 e = low[q];
        const int code = __float_as_int(e.w);
        const bool is_near = code >= 0 && (unsigned)((code & 0xffff) - ppx) < RD_NEAR_W &&
                             (unsigned)((code >> 16) - r0) < RD_NEAR_ROWS;
        // least and largest lateral distances to the panel's points
        const float ux = fabsf(e.x - ox), uy = fabsf(e.y - oy), z2 = fmaf(e.z, e.z, 1e-20f);
        const float bx = fmaxf(ux - ax, 0.0f), by = fmaxf(uy - ay, 0.0f), tx = ux + ax, ty = uy + ay;
        const float inv = rsqrtf(fmaf(bx, bx, fmaf(by, by, z2)));
        const float i2 = inv * inv, v7 = is_near ? 0.0f : (e.z * inv) * (i2 * i2 * i2);
        // c_x^2 <= 0.68 over the panel: 0.32 x^2 <= 0.68 (y^2 + z^2)
        Tx = fmaf(0.32f * tx * tx <= 0.68f * fmaf(by, by, z2) ? 2.5f : 15.0f, v7, Tx);
        Ty = fmaf(0.32f * ty * ty <= 0.68f * fmaf(bx, bx, z2) ? 2.5f : 15.0f, v7, Ty);
      }
      here = 0;
      __syncthreads();
      if (tid == 0) s_n = 0;
      __syncthreads();
    }
    for (int o = 16; o > 0; o >>= 1) {
      Tx += __shfl_xor_sync(0xffffffffu, Tx, o);
      Ty += __shfl_xor_sync(0xffffffffu, Ty, o);
      gT += __shfl_xor_sync(0xffffffffu, gT, o);
    }
    if (lane == 0) s_gT[tid >> 5] = gT;
    __syncthreads();
    gT = 0.0f;
    for (int q = 0; q < 8; ++q) gT += s_gT[q];
    __syncthreads();
    Tx = fmaf(15.0f, gT, Tx);
    Ty = fmaf(15.0f, gT, Ty);
    if (!live) continue;   // (at the end of the item's work: no barrier is left)
    float* rec = nr.rec + (size_t)(p.q_off / 16 + pan) * RD_NEAR_REC;
    if (lane < 16) rec[lane] = c;
    // the rows of near electrons end to end: what turns a list index into an electron, and the row's end
    int a0 = 0, len = 0;
    if (lane < RD_NEAR_ROWS) {
      const int row = (r0 + lane) * nb + ppx;
      a0 = start[row];
      len = start[row + RD_NEAR_W] - a0;
    }
    int end = len;
    for (int o = 1; o < RD_NEAR_ROWS; o <<= 1) {
      const int v2 = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v2;
    }
    if (lane < RD_NEAR_ROWS) {
      reinterpret_cast<int*>(rec)[20 + lane] = end;
      reinterpret_cast<int*>(rec)[20 + RD_NEAR_ROWS + lane] = a0 - (end - len);
    }
    if (lane == 0) *reinterpret_cast<float4*>(rec + 16) = make_float4(ox, oy, 1.03f * Tx, big);
    if (lane == 1) *reinterpret_cast<float2*>(rec + 28) = make_float2(1.03f * Ty, RD_U24 * rd_near_units(NP, cnt));
  }
}

// Bound on |estimate - pair sum| at (tx, ty) of a panel: the interpolation's
// error, and the roundings of the pair sum (153 u of the sum of magnitudes A at
// the point, the same of the nodes' `big` carried through the interpolation),
// of the near sums (a run of 32 terms, the lanes' sums, and one more addition for
// every further run: rd_bounds.h, which k_near_panels has put into `big` and the
// record's last word), of the points' own coordinates (half
// an ulp of the emitter's half width, against the distance 5 a to the nearest
// far electron: 0.6 P u) and of the evaluation (~30 u).
// near_bound0 is the part that does not depend on A (factor: the record's last word).
__device__ __forceinline__ float near_bound0(const DiodeParams& p, float tx, float ty, float Tx, float Ty, float big) {
  const float x2 = tx * tx, y2 = ty * ty;
  const float wx = fabsf((x2 - 0.741555748f) * (x2 - 0.115587109f)), wy = fabsf((y2 - 0.741555748f) * (y2 - 0.115587109f));
  const float lx = 1.48f + 14.0f * fmaxf(fabsf(tx) - 0.9f, 0.0f), ly = 1.48f + 14.0f * fmaxf(fabsf(ty) - 0.9f, 0.0f);
  const float ax2 = p.nr_ax * p.nr_ax, ay2 = p.nr_ay * p.nr_ay;
  return Tx * ((wx + 1e-5f) * (ax2 * ax2)) + Ty * (lx * (wy + 1e-5f) * (ay2 * ay2)) +
         RD_U24 * (lx * ly * rd_near_units(p.nr_P, 0) * big);
}

// The pair sums of k_mh_jump_planar at two points, by the NT threads of a block,
// bit for bit.  A warp takes two j-tiles at a time: its lanes form the factors
// 1/r^3 of both points (the part that can run in parallel), four lanes add them up,
// one (tile, point) each, in the tile kernel's order from zero; then the tile sums
// of a chunk are folded in order with two-sum and the chunks added in order with
// pair_add (pair_partials).  out[0], out[1]: the sums before z0_finish.
// 4800 electrons: ~3 us (40 us with one thread per tile, whose strided loads and
// reciprocal roots all sit on the sum's chain).
#define RD_NEAR_PASS 128      // tiles per pass over the electrons
template <int NT>
struct NearExact {
  float4 f[NT / 32][2][2][RD_TILE / 4];   // 1/r^3 of (tile, point), by warp
  float4 q[NT / 32][2][RD_TILE / 4];      // q z of the tile
  float t[2][RD_NEAR_PASS];
  float h[2][RD_NCH_MAX], l[2][RD_NCH_MAX];
  double out[2];
  int still;
};
template <int NT>
__device__ __forceinline__ void near_exact2(const float4* __restrict__ zhi, const float4* __restrict__ zlo, int n,
                                            int clen, int nch, float x0, float y0, float x1, float y1,
                                            NearExact<NT>* s) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int tiles = (n + RD_TILE - 1) / RD_TILE, tpc = clen / RD_TILE;
  float ch = 0.0f, cl = 0.0f;   // the open chunk of point tid (threads 0 and 1)
  int in_chunk = 0, chunk = 0;
  for (int base = 0; base < tiles; base += RD_NEAR_PASS) {
    const int here = min(RD_NEAR_PASS, tiles - base);
    for (int t2 = 2 * w; t2 < here; t2 += NT / 16) {
      float4 h[2][RD_TILE / 32];
      float2 l[2][RD_TILE / 32];
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int v = 0; v < RD_TILE / 32; ++v) {   // all loads in flight; past the electrons q z = 0
          const int j = (base + t2 + b) * RD_TILE + lane + 32 * v;
          h[b][v] = j < n ? zhi[j] : make_float4(0.0f, 0.0f, 1.0f, 0.0f);
          l[b][v] = j < n ? *reinterpret_cast<const float2*>(&zlo[j]) : make_float2(0.0f, 0.0f);
        }
#pragma unroll
      for (int b = 0; b < 2; ++b)
#pragma unroll
        for (int v = 0; v < RD_TILE / 32; ++v) {
          const int k = lane + 32 * v;
          const float dx0 = (x0 - h[b][v].x) - l[b][v].x, dy0 = (y0 - h[b][v].y) - l[b][v].y;
          const float dx1 = (x1 - h[b][v].x) - l[b][v].x, dy1 = (y1 - h[b][v].y) - l[b][v].y;
          const float i0 = rsqrtf(fmaf(dx0, dx0, fmaf(dy0, dy0, h[b][v].z)));
          const float i1 = rsqrtf(fmaf(dx1, dx1, fmaf(dy1, dy1, h[b][v].z)));
          reinterpret_cast<float*>(s->q[w][b])[k] = h[b][v].w;
          reinterpret_cast<float*>(s->f[w][b][0])[k] = (i0 * i0) * i0;
          reinterpret_cast<float*>(s->f[w][b][1])[k] = (i1 * i1) * i1;
        }
      __syncwarp();
      if (lane < 4 && t2 + (lane >> 1) < here) {   // a term with q z = 0 adds nothing
        const int b = lane >> 1, pt = lane & 1;
        float a = 0.0f;
#pragma unroll 8
        for (int k = 0; k < RD_TILE / 4; ++k) {
          const float4 q = s->q[w][b][k], f = s->f[w][b][pt][k];
          a = fmaf(q.x, f.x, a);
          a = fmaf(q.y, f.y, a);
          a = fmaf(q.z, f.z, a);
          a = fmaf(q.w, f.w, a);
        }
        s->t[pt][t2 + b] = a;
      }
      __syncwarp();
    }
    __syncthreads();
    if (tid < 2) {   // RD_NEAR_PASS need not hold whole chunks: the open one carries over
      for (int i = 0; i < here; ++i) {
        two_sum_acc(ch, cl, s->t[tid][i]);
        if (++in_chunk == tpc || base + i + 1 == tiles) {
          s->h[tid][chunk] = ch;
          s->l[tid][chunk] = cl;
          ch = cl = 0.0f;
          in_chunk = 0;
          ++chunk;
        }
      }
    }
    if (base + RD_NEAR_PASS < tiles) __syncthreads();
  }
  if (tid < 2) {
    float H = 0.0f, L = 0.0f;
    if (tiles > 0 && nch == 1) {
      H = s->h[tid][0];
      L = s->l[tid][0];
    } else {
      for (int c = 0; c < nch && tiles > 0; ++c) pair_add(H, L, s->h[tid][c], s->l[tid][c]);
    }
    s->out[tid] = (double)H + (double)L;
  }
  __syncthreads();
}

// The decision of mh_decide_f from estimated fields: the proposal's Fn within dF of
// the pair sum's, the chain's Fc within fe; t0, t2 the proposal's work-function
// entry, lu the accept test's log u.  The fields' errors widen the guard: each
// relative error is at most 1/4 and enters 2 log(-F) - rho at most 2.5-fold.
// Returns 1 taken, 0 rejected, -1 open; *rn the proposal's rho (if taken).
__device__ __forceinline__ int near_decide(const DiodeParams& p, float Fn, float dF, float Fc, float fe, float rc,
                                           float t0, float t2, float lu, float* rn) {
  if (Fn - dF > 0.0f) return 0;   // F >= 0: rejected
  if (!(Fn < 0.0f && 4.0f * dF <= -Fn)) return -1;
  *rn = rho_entry_f(p, t0, t2, Fn);
  const float l2 = 2.0f * logf(Fn / Fc), df = l2 - (*rn - rc);
  const float St = fabsf(l2) + fabsf(*rn) + fabsf(rc);
  const float eps = 2.5f * (dF / -Fn + fe / -Fc);
  if (!(isfinite(df) && isfinite(eps) && isfinite(lu))) return -1;
  const float gd = rd_near_guard(St + fabsf(lu)) + eps;
  if (df >= rd_near_guard(St) + eps || lu <= df - gd) return 1;
  return lu > df + gd ? 0 : -1;
}

// Field from a sum, and the rounding of that step.
__device__ __forceinline__ float near_field(const DiodeParams& p, float ksc, float S, float dS, float* dF) {
  const float A0 = -2.0f * ksc;
  *dF = fabsf(A0) * dS + 2.4e-7f * (fabsf(p.nr_Ez) + fabsf(A0 * S));
  return fmaf(A0, S, p.nr_Ez);
}

// A jump that the interpolated estimate leaves open (rare; out of line so that it
// costs the others no registers).  First the direct sums at the proposal (px, py)
// and at the chain's point (cx, cy) by the whole block, in any order: they lie
// within the roundings of the two sums (153 u for the pair sum, 25 u a term and the
// order here: rd_near_direct_units) of the pair sums, some twenty times closer than the
// estimate, and let the targets be compared in FP64; what even they leave open takes
// the pair sums (near_exact2) and
// mh_accept_one_f's test.  The thread that holds the chain (mine) decides and
// updates it; returns 1 there if the proposal is taken.
template <int NT>
__device__ __noinline__ int near_open(const DiodeParams& p, const Pool& pool, const ChainState& cs,
                                      const double* __restrict__ wtab, const PlanEntry& e, double kscale, bool mine,
                                      int c, int k, int it_idx, uint32_t step, float px, float py, float cx, float cy,
                                      float lu, NearExact<NT>* s) {
  const float4* zhi = pool.zk_hi + p.off;
  const float4* zlo = pool.zk_lo + p.off;
  const int n = e.n_j, tid = threadIdx.x;
  float sn = 0.0f, sc = 0.0f, rn = 0.0f, rc = 0.0f;
  for (int j0 = 0; j0 < n; j0 += 8 * NT) {   // eight loads in flight, runs of eight terms
    float4 h[8];
    float2 l[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int j = j0 + q * NT + tid;
      h[q] = j < n ? zhi[j] : make_float4(0.0f, 0.0f, 1.0f, 0.0f);
      l[q] = j < n ? *reinterpret_cast<const float2*>(&zlo[j]) : make_float2(0.0f, 0.0f);
    }
    rn = rc = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q) { rn += near_term(h[q], l[q], px, py); rc += near_term(h[q], l[q], cx, cy); }
    sn += rn;
    sc += rc;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sn += __shfl_xor_sync(0xffffffffu, sn, o);
    sc += __shfl_xor_sync(0xffffffffu, sc, o);
  }
  if ((tid & 31) == 0) { s->t[0][tid >> 5] = sn; s->t[1][tid >> 5] = sc; }
  if (tid == 0) s->still = 0;
  __syncthreads();
  int a = 0;
  if (mine) {
    sn = sc = 0.0f;
    for (int w = 0; w < NT / 32; ++w) { sn += s->t[0][w]; sc += s->t[1][w]; }
    const float eu = RD_U24 * rd_near_direct_units(n, NT);
    float dFn, dFc, t0, t2, r;
    const float Fn = near_field(p, (float)kscale, sn, eu * fabsf(sn), &dFn);
    work_entry_f(p, wtab, chain_cell_f(p, px, py), px, py, &t0, &t2);
    float Fc = cs.fF[k], fe = cs.fe[k], rho = cs.fsup[k];
    if (fe != 0.0f) {
      const float F2 = near_field(p, (float)kscale, sc, eu * fabsf(sc), &dFc);
      if (dFc < fe && F2 < 0.0f && 4.0f * dFc <= -F2) {
        Fc = F2; fe = dFc;
        rho = rho_xy_f(p, wtab, cx, cy, F2);
        cs.fF[k] = Fc; cs.fe[k] = fe; cs.fsup[k] = rho;
      }
    }
    int take = near_decide(p, Fn, dFn, Fc, fe, rho, t0, t2, lu, &r);
    const double Dn = p.E_z - 2.0 * kscale * (double)sn, Dc = p.E_z - 2.0 * kscale * (double)sc;
    if (take < 0 && Dn < 0.0 && Dc < 0.0) {   // the targets in FP64: only the sums' own bounds remain
      const double en = 2.0 * kscale * (double)eu * fabs((double)sn), ec = 2.0 * kscale * (double)eu * fabs((double)sc);
      if (4.0 * en <= -Dn && 4.0 * ec <= -Dc) {
        uint32_t o[4];
        philox4x32((uint32_t)c, (uint32_t)it_idx, step, RNG_ACCEPT, (uint32_t)p.seed, (uint32_t)(p.seed >> 32), o);
        const double d = (supply_log_chain_d(p, wtab, px, py, Dn) - supply_log_chain_d(p, wtab, cx, cy, Dc)) -
                         log(u01_words(o[0], o[1]));
        const double eps = 2.5 * (en / -Dn + ec / -Dc) + 1.0e-11;   // take iff d >= 0 (or s_n >= s_c, where log u <= 0)
        if (d > eps) take = 1;
        else if (d < -eps) take = 0;
        r = rho_entry_f(p, t0, t2, Fn);
      }
    }
    if (take == 1) {
      cs.fx[k] = px; cs.fy[k] = py; cs.fsup[k] = r; cs.fF[k] = Fn; cs.fe[k] = dFn;
      a = 1;
    }
    s->still = take < 0;
  }
  __syncthreads();
  if (!s->still) return a;   // block-uniform
  near_exact2<NT>(zhi, zlo, n, e.clen, e.nch, px, py, cx, cy, s);
  if (mine) {
    const double F = z0_finish<1>(p, s->out[0], kscale);
    if (cs.fe[k] != 0.0f) {   // the current point's field was an estimate
      const double Fc = z0_finish<1>(p, s->out[1], kscale);
      const float Fcf = (float)Fc;
      cs.F[k] = Fc; cs.fF[k] = Fcf; cs.fe[k] = 0.0f;
      cs.fsup[k] = rho_xy_f(p, wtab, cx, cy, Fcf);
    }
    if (F < 0.0) {
      const float Ff = (float)F;
      const float r = rho_xy_f(p, wtab, px, py, Ff);
      if (mh_decide_f(p, wtab, c, it_idx, step, F, Ff, r, px, py, cx, cy, cs.F[k], cs.fF[k], cs.fsup[k])) {
        cs.fx[k] = px; cs.fy[k] = py; cs.fsup[k] = r; cs.fF[k] = Ff; cs.F[k] = F; cs.fe[k] = 0.0f;
        a = 1;
      }
    }
  }
  __syncthreads();
  return a;
}

// The FP64 chains' open jumps, in the two stages of near_open.  First FP64 sums at both
// points by the block in any order: with nt threads they lie within n / nt + 200
// additions' and 8 terms' roundings (v = 2^-53) of the pair sums, and compare the targets
// to 1e-11.  What even they leave open takes the pair sums of k_mh_jump_planar bit for bit
// -- a thread per point and tile, the tiles of a chunk and then the chunks in order -- and
// the test of mh_accept_one.  A point whose field is a pair sum already (fe = 0) keeps it,
// and its target.  1200 electrons: 2 us an open jump, 25 us with the pair sums at once.
template <int NT>
struct NearExact64 {
  double t[2][NT / 2];   // a pass's tile sums
  double out[2];
  int still;
};
template <int NT>
__device__ __noinline__ void near_exact64(const DiodeParams& p, const Pool& pool, const PlanEntry& e, double px,
                                          double py, double cx, double cy, NearExact64<NT>* s) {
  const int tid = threadIdx.x, n = e.n_j, tiles = (n + RD_TILE - 1) / RD_TILE, tpc = e.clen / RD_TILE;
  const float L2x3 = (float)(3.0 * c_k.L2);
  const int q = tid / (NT / 2), slot = tid % (NT / 2);
  const double x = q ? cx : px, y = q ? cy : py;
  double chunk = 0.0, all = 0.0;   // threads 0 and 1: a point each
  int in_chunk = 0;
  for (int base = 0; base < tiles; base += NT / 2) {
    const int j0 = (base + slot) * RD_TILE;
    double a = 0.0;
#pragma unroll 4
    for (int j = j0; j < min(j0 + RD_TILE, n); ++j) {
      const int g = p.off + j;
      a = z0_add_f64(a, make_d4(pool.x[g], pool.y[g], pool.z[g], pool.q[g]), x, y, 0, p.d, c_k.L2, L2x3);
    }
    s->t[q][slot] = a;
    __syncthreads();
    if (tid < 2)
      for (int i = 0; i < min(NT / 2, tiles - base); ++i) {
        chunk += s->t[tid][i];
        if (++in_chunk == tpc || base + i + 1 == tiles) {
          all = e.nch > 1 ? all + chunk : chunk;
          chunk = 0.0;
          in_chunk = 0;
        }
      }
    __syncthreads();
  }
  if (tid < 2) s->out[tid] = all;
  __syncthreads();
}

template <int NT>
__device__ __noinline__ int near_open64(const DiodeParams& p, const Pool& pool, const ChainState& cs,
                                        const double* __restrict__ wtab, const PlanEntry& e, double kscale, bool mine,
                                        int c, int k, int it_idx, uint32_t step, double px, double py, double cx,
                                        double cy, NearExact64<NT>* s) {
  const int tid = threadIdx.x, n = e.n_j;
  const float L2x3 = (float)(3.0 * c_k.L2);
  double s0 = 0.0, s1 = 0.0;
  for (int j = tid; j < n; j += NT) {
    const int g = p.off + j;
    const rd_d4 pj = make_d4(pool.x[g], pool.y[g], pool.z[g], pool.q[g]);
    s0 = z0_add_f64(s0, pj, px, py, 0, p.d, c_k.L2, L2x3);
    s1 = z0_add_f64(s1, pj, cx, cy, 0, p.d, c_k.L2, L2x3);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
  if ((tid & 31) == 0) { s->t[0][tid >> 5] = s0; s->t[1][tid >> 5] = s1; }
  __syncthreads();
  int a = 0;
  float t0, t2;
  double lu = 0.0;
  if (mine) {
    s0 = s1 = 0.0;
    for (int w = 0; w < NT / 32; ++w) { s0 += s->t[0][w]; s1 += s->t[1][w]; }
    const double v = 1.12e-16 * (n / NT + 208), E = fabs(p.E_z);
    const bool exact = cs.fe[k] == 0.0f;
    const double F = z0_finish<0>(p, s0, kscale), Fc = exact ? cs.F[k] : z0_finish<0>(p, s1, kscale);
    const double en = v * (fabs(F) + 2.0 * E), ec = exact ? 0.0 : v * (fabs(Fc) + 2.0 * E);   // |S| <= |F| + |E|
    double u1, u2;
    rng2(p.seed, (uint32_t)c, (uint32_t)it_idx, step, RNG_ACCEPT, &u1, &u2);
    lu = log(u1);
    int take = F > en ? 0 : -1;
    if (F < 0.0 && Fc < 0.0 && 4.0 * en <= -F && 4.0 * ec <= -Fc) {
      const double sc = exact ? cs.sup[k] : supply_log_xy(p, wtab, cx, cy, Fc);
      const double d = (supply_log_xy(p, wtab, px, py, F) - sc) - lu;
      const double eps = 2.5 * (en / -F + ec / -Fc) + 1.0e-11;   // take iff d >= 0 (log u <= 0)
      take = d > eps ? 1 : d < -eps ? 0 : -1;
    }
    if (!exact) {
      work_entry_d(p, wtab, cx, cy, &t0, &t2);
      cs.fF[k] = (float)Fc;
      cs.fe[k] = 1.2e-7f * fabsf((float)Fc);
      cs.fsup[k] = rho_entry_f(p, t0, t2, (float)Fc);
    }
    if (take == 1) {
      work_entry_d(p, wtab, px, py, &t0, &t2);
      cs.x[k] = px; cs.y[k] = py;
      cs.fF[k] = (float)F;
      cs.fe[k] = 1.2e-7f * fabsf((float)F);
      cs.fsup[k] = rho_entry_f(p, t0, t2, (float)F);
      a = 1;
    }
    s->still = take < 0;
  }
  __syncthreads();
  const int still = s->still;
  __syncthreads();   // (read before the next call writes it)
  if (!still) return a;   // block-uniform
  near_exact64<NT>(p, pool, e, px, py, cx, cy, s);
  if (mine) {
    if (cs.fe[k] != 0.0f) {   // the chain's field was an estimate
      const double Fc = z0_finish<0>(p, s->out[1], kscale);
      cs.F[k] = Fc;
      cs.sup[k] = supply_log_xy(p, wtab, cx, cy, Fc);
      cs.fF[k] = (float)Fc;
      cs.fe[k] = 0.0f;
    }
    const double F = z0_finish<0>(p, s->out[0], kscale);
    if (F < 0.0) {
      const double sn = supply_log_xy(p, wtab, px, py, F), sc = cs.sup[k];
      if (sn >= sc || lu <= sn - sc) {
        work_entry_d(p, wtab, px, py, &t0, &t2);
        cs.x[k] = px; cs.y[k] = py;
        cs.F[k] = F; cs.sup[k] = sn;
        cs.fF[k] = (float)F;
        cs.fe[k] = 0.0f;
        cs.fsup[k] = rho_entry_f(p, t0, t2, (float)F);
        a = 1;
      }
    }
  }
  __syncthreads();
  return a;
}

// The plan entry of item g: two rounds of 32 slots each instead of a binary search's
// chain of loads (more than 1024 slots take decode_item).
__device__ __forceinline__ int near_entry(const PlanEntry* __restrict__ plan, int nd, int g, int lane) {
  if (nd == 1) return 0;
  if (nd > 1024) return decode_item(plan, nd, g).d;
  const int step = (nd + 31) / 32;
  const int i = lane * step;
  const int seg = __popc(__ballot_sync(0xffffffffu, i < nd && plan[i].item_off <= g)) - 1;
  const int j = seg * step + lane;
  return seg * step + __popc(__ballot_sync(0xffffffffu, lane < step && j < nd && plan[j].item_off <= g)) - 1;
}

// The acceptance counts of one tile, after the warm-up (whose step size is fixed: its
// jumps neither count nor wait); the diode's last tile updates MH_std
// (MH_std_update :603-612, as mh_std_step) and lets the next jump go.  One packed
// atomic carries the tile count and both sums, so its answer tells the last tile
// the diode's totals.  At the upper clamp with a rate above 0.35 the product stays
// clamped, whatever the factor: no FP64 exponential on the jump's critical path;
// the rate itself is only kept at the last jump (every jump counts the same chains).
__device__ __forceinline__ void near_counts(const DiodeParams& p, DiodeDyn& y, unsigned long long* count,
                                            unsigned long long* progress, unsigned long long last, int tiles, int it_idx,
                                            int a, int r) {
  const unsigned long long add = (1ull << 44) | ((unsigned long long)a << 22) | (unsigned long long)r;
  const unsigned long long now = atomicAdd(count, add) + add;
  if ((int)(now >> 44) != tiles) return;
  __stcg(count, 0ull);
  const int A = (int)(now >> 22) & 0x3fffff, R = (int)now & 0x3fffff;
  unsigned long long next = (last & ~0x7fffffffull) | (unsigned)it_idx;   // the step size stays
  if (A + R > 0 &&
      (it_idx == p.mh_jumps || !((unsigned)last & RD_NEAR_CLAMPED) || 20ll * A <= 7ll * (A + R))) {
    const double g = mh_std_gain(A, R, &y.a_rate);
    const double m = mh_std_clamp(p, __ldcg(&y.MH_std) * g);
    __stcg(&y.MH_std, m);
    next = near_progress(p, it_idx, m);
  }
  __threadfence();
  *reinterpret_cast<volatile unsigned long long*>(progress) = next;
}

// A lone diode's form of near_counts without a second hop: jump it's tiles add to ring
// word it & 3, every block reads the words itself and forms the same step size from
// them.  A word is cleared two jumps before its next use by the block of the diode's
// first tile, which then knows that every block has read it (all of them have counted
// in the jump after).  Returns false if the wait gave up.  Without the fence and the
// second word a jump of 121 blocks takes 0.1 us less (FP32, 4.5 us) and 1.6 us less
// (FP64, whose step size was read from memory, 8.7 us); 1.6 us from the last block's
// count to the last block's start are left.
__device__ __forceinline__ bool near_wait_counts(const unsigned long long* word, int tiles, int* A, int* R) {
  const volatile unsigned long long* v = word;
  unsigned long long now = *v;
  for (int spins = 0; (int)(now >> 44) != tiles && spins < RD_NEAR_SPIN; ++spins) now = *v;
  *A = (int)(now >> 22) & 0x3fffff;
  *R = (int)now & 0x3fffff;
  return (int)(now >> 44) == tiles;
}

// Every jump of every chain of the diodes with the near / far split, in one
// cooperative launch.  A block of NW warps takes 32 chains at a time (an item of the
// PM_MH_NEAR plan) through a jump: warp 0 proposes and evaluates the far part, one
// chain per lane, while other warps draw log u and the next Gaussian pairs; every
// chain's near electrons are summed by eight lanes (loads of four electrons in
// flight per lane); warp 0 decides; the jumps left open take the pair sums
// (near_open).  A jump needs the acceptance counts of the whole diode's last one
// (MH_std), nothing of any other diode: a block walks its items jump by jump and
// waits only for the diode's progress word.  All blocks are resident (cooperative
// launch) and an item waits only for items of earlier jumps, so every wait ends;
// each still polls at most RD_NEAR_SPIN times (about a second), after which the
// block counts in *gave_up and leaves (rd_run reports it).
// ONE: every block has at most one item; its chains stay in registers.
template <int PREC, int NW>
struct NearShared {
  using Real = typename std::conditional<PREC == 1, float, double>::type;
  float x[32], y[32], near[32], lu[32];   // proposal (nm; FP64 chains: high words), near sum, log u
  float xl[PREC == 1 ? 1 : 32], yl[PREC == 1 ? 1 : 32];   // FP64 chains: low words
  float wide[PREC == 1 ? 1 : 32];                         // and how far the near sum may be off (near_wide)
  Real g[2][32];                          // next Gaussian pair
  int pan[32];                            // the chain's panel; -1: no chain
  Real ox[32], oy[32], cx[32], cy[32];    // proposals and chains' points, where a jump is left open
  unsigned open;
  int dead;
  typename std::conditional<PREC == 1, NearExact<32 * NW>, NearExact64<32 * NW>>::type ex;
};

template <int PREC>
__device__ __forceinline__ typename std::conditional<PREC == 1, float, double>::type* near_sel(float* f, double* d) {
  if constexpr (PREC == 1) return f; else return d;
}

// The far part at a point: a panel's record, then its value and bound (c0.x, c0.y).
struct NearFar {
  float4 c0, c1, c2, c3, cm;
  float2 ty;   // and the rounding per |S|
  __device__ __forceinline__ void load(const float4* rec) {
    c0 = rec[0]; c1 = rec[1]; c2 = rec[2]; c3 = rec[3]; cm = rec[4];
    ty = reinterpret_cast<const float2*>(rec)[14];
  }
  __device__ __forceinline__ void eval(const DiodeParams& p, float px, float py) {
    const float x = (px - cm.x) * p.nr_iax, y = (py - cm.y) * p.nr_iay;
    const float r0 = fmaf(fmaf(fmaf(c0.w, x, c0.z), x, c0.y), x, c0.x);
    const float r1 = fmaf(fmaf(fmaf(c1.w, x, c1.z), x, c1.y), x, c1.x);
    const float r2 = fmaf(fmaf(fmaf(c2.w, x, c2.z), x, c2.y), x, c2.x);
    const float r3 = fmaf(fmaf(fmaf(c3.w, x, c3.z), x, c3.y), x, c3.x);
    c0.y = near_bound0(p, x, y, cm.z, ty.x, cm.w);
    c0.x = fmaf(fmaf(fmaf(r3, y, r2), y, r1), y, r0);
  }
};

template <int PREC, int NW, bool ONE>
__device__ __forceinline__ void near_jumps(NearShared<PREC, NW>& sh, const DiodeParams* __restrict__ P,
                                           DiodeDyn* __restrict__ Dy, const Pool& pool, const PlanEntry* __restrict__ plan, int total, int nd,
                                           const PlanEntry* __restrict__ plan_mh, const ChainState& cs,
                                           const int* __restrict__ ch_off, const double* __restrict__ wtab,
                                           int engine_step, int jumps, const NearState& nr, double kscale, int* gave_up) {
  using Real = typename NearShared<PREC, NW>::Real;
  constexpr int NT = 32 * NW, ROUNDS = 8 / NW;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (tid == 0) sh.dead = 0;
  const float ksc = (float)kscale;
  // the chains' points and Gaussian pairs in memory: nm from the emitter's centre, or m
  Real* const ax = near_sel<PREC>(cs.fx, cs.x);
  Real* const ay = near_sel<PREC>(cs.fy, cs.y);
  Real* const agx = near_sel<PREC>(cs.fgx, cs.gx);
  Real* const agy = near_sel<PREC>(cs.fgy, cs.gy);
  // the chains of the block's item (ONE; warp 0)
  Real fx = 0, fy = 0, gx = 0, gy = 0;
  float Fc = 0.0f, rc = 0.0f, fe = 0.0f;
  double std_ = 0.0;   // (ONE) the step size
  int ok = 0, d = 0;
  for (int it = 1; it <= jumps; ++it) {
    for (int g = blockIdx.x; g < total; g += gridDim.x) {
      if (!ONE || it == 1) d = near_entry(plan, nd, g, lane);
      const DiodeParams& p = P[d];
      if (it > p.mh_jumps) continue;
      DiodeDyn& y = Dy[d];
      const int ndim_first = (p.mh_jumps + 2) / 4;   // nint(0.25 mh_jumps), :1141
      const int M = plan[d].n_i, c = (g - plan[d].item_off) * 32 + lane, k = ch_off[d] + c;
      const uint32_t step = (uint32_t)(engine_step - y.step_offset);
      const float* recs = nr.rec + (size_t)(p.q_off / 16) * RD_NEAR_REC;
      float px = 0.0f, py = 0.0f, t0 = 0.0f, t2 = 0.0f;
      bool off = false;      // no panel's expansion holds there
      Real ox = 0, oy = 0;   // the proposal
      NearFar far_part;
      unsigned long long pr = 0;
      if (NW > 1 ? w == NW - 1 : true) {   // the next proposal's Gaussian pair
        if (c < M && it < p.mh_jumps && cs.ok[k]) {
          Real g1, g2;
          if constexpr (PREC == 1) gauss2f(p.seed, (uint32_t)c, (uint32_t)(it + 1), step, &g1, &g2);
          else gauss2(p.seed, (uint32_t)c, (uint32_t)(it + 1), step, &g1, &g2);
          sh.g[0][lane] = g1;
          sh.g[1][lane] = g2;
        }
      }
      if (w == (NW > 1 ? 1 : 0) && c < M) {   // log u of the accept test, as mh_decide_f forms it
        uint32_t o[4];
        philox4x32((uint32_t)c, (uint32_t)it, step, RNG_ACCEPT, (uint32_t)p.seed, (uint32_t)(p.seed >> 32), o);
        sh.lu[lane] = logf(fmaf((float)(o[1] >> 11), 1.1102230246251565e-16f, (float)o[0] * 2.3283064365386963e-10f));
      }
      if (w == 0) {
        if (!ONE || it == 1) {
          ok = c < M ? cs.ok[k] : 0;
          if (ok) {
            fx = ax[k]; fy = ay[k]; gx = agx[k]; gy = agy[k];
            Fc = cs.fF[k]; rc = cs.fsup[k]; fe = cs.fe[k];
          }
        }
        // the step size: fixed during the warm-up jumps, then MH_std after the last jump
        if (ONE) {
          if (lane == 0) {
            if (it == 1) {
              std_ = __ldcg(&y.MH_std);
            } else if (it - 1 > ndim_first) {
              int A, R;
              if (!near_wait_counts(nr.ring + 4 * d + ((it - 1) & 3), plan[d].tiles, &A, &R)) sh.dead = 1;
              double rate;
              if (A + R > 0 && (std_ != p.mh_hi || 20ll * A <= 7ll * (A + R)))
                std_ = mh_std_clamp(p, std_ * mh_std_gain(A, R, &rate));
            }
          }
          std_ = __shfl_sync(0xffffffffu, std_, 0);
        } else {
          if (lane == 0) {
            const volatile unsigned long long* prog = nr.progress + d;
            pr = *prog;
            const int need = it - 1 > ndim_first ? it - 1 : 0;   // the warm-up's step size is fixed: no wait
            for (int spins = 0; (int)((unsigned)pr & ~RD_NEAR_CLAMPED) < need && spins < RD_NEAR_SPIN; ++spins) pr = *prog;
            if ((int)((unsigned)pr & ~RD_NEAR_CLAMPED) < need) sh.dead = 1;
          }
          pr = __shfl_sync(0xffffffffu, pr, 0);
        }
        if constexpr (PREC == 1) {   // mh_propose_f32
          const float mhs = ONE ? (float)std_ : __uint_as_float((unsigned)(pr >> 32));
          const float sx = (it > ndim_first) ? p.em_wx * mhs : p.em_wx * 0.10f;
          const float sy = (it > ndim_first) ? p.em_wy * mhs : p.em_wy * 0.10f;
          if (ok) {
            const float hx = p.em_hx, hy = p.em_hy;
            px = fmaf(gx, sx, fx);
            py = fmaf(gy, sy, fy);
            if (px > hx) px = hx - (px - hx); else if (px < -hx) px = -hx - (px + hx);
            if (py > hy) py = hy - (py - hy); else if (py < -hy) py = -hy - (py + hy);
          }
          ox = px; oy = py;
        } else {                     // mh_propose_f64
          if (!ONE) __threadfence();   // MH_std was written before the progress word
          const double mhs = ONE ? std_ : __ldcg(&y.MH_std);
          const double sx = (it > ndim_first) ? p.em_Lx * mhs : p.em_Lx * 0.10;
          const double sy = (it > ndim_first) ? p.em_Ly * mhs : p.em_Ly * 0.10;
          ox = p.em_x0; oy = p.em_y0;
          if (ok) {
            const double hx = p.em_x0 + p.em_Lx, hy = p.em_y0 + p.em_Ly;
            ox = fma(gx, sx, fx);
            oy = fma(gy, sy, fy);
            if (ox > hx) ox = hx - (ox - hx); else if (ox < p.em_x0) ox = (p.em_x0 - ox) + p.em_x0;
            if (oy > hy) oy = hy - (oy - hy); else if (oy < p.em_y0) oy = (p.em_y0 - oy) + p.em_y0;
          }
          float lx, ly;
          split_nm(ox, p.org_x, &px, &lx);
          split_nm(oy, p.org_y, &py, &ly);
          sh.xl[lane] = lx; sh.yl[lane] = ly;
        }
        const int NP = p.nr_P;
        const int ppx = min(max((int)floorf((px + p.em_hx) * p.nr_iwx), 0), NP - 1);
        const int ppy = min(max((int)floorf((py + p.em_hy) * p.nr_iwy), 0), NP - 1);
        const int pan = ppy * NP + ppx;
        sh.x[lane] = px; sh.y[lane] = py;
        sh.pan[lane] = ok ? pan : -1;
        if (NW > 1) __syncthreads(); else __syncwarp();
        const float4* rec = reinterpret_cast<const float4*>(recs + (size_t)pan * RD_NEAR_REC);
        far_part.load(rec);
        if (!ONE) far_part.eval(p, px, py);   // (ONE: evaluated after the near sums, the loads in flight meanwhile)
        // a step size above the clamp (from a checkpoint) can reflect a proposal off the emitter
        off = fmaxf(fabsf(px) - p.em_hx, fabsf(py) - p.em_hy) > 0.005f * fminf(p.nr_ax, p.nr_ay);
        if (ok) {
          if constexpr (PREC == 1) work_entry_f(p, wtab, chain_cell_f(p, px, py), px, py, &t0, &t2);
          else work_entry_d(p, wtab, ox, oy, &t0, &t2);
        }
      } else {
        __syncthreads();
      }
      if (sh.dead) {   // block-uniform
        if (tid == 0) atomicAdd(gave_up, 1);
        return;
      }
      if (ONE && tid == NT - 32 && it > ndim_first && g == plan[d].item_off) {   // the word of jump it + 2 (a barrier before this jump's count)
        __stcg(nr.ring + 4 * d + ((it + 2) & 3), 0ull);
        __threadfence();
      }
      // near electrons
      for (int r8 = 0; r8 < ROUNDS; ++r8) {
        const int l = lane & 7, q = (w * ROUNDS + r8) * 4 + (lane >> 3), pan = sh.pan[q];
        float s = 0.0f, wide = 0.0f;
        if (pan >= 0) {
          const float kw = near_wide(p);
          // the list's rows: their ends in it, and what turns an index of it into an electron
          const int4* rt = reinterpret_cast<const int4*>(recs + (size_t)pan * RD_NEAR_REC + 20);
          const int4 end = rt[0], at = rt[1];
          const float x = sh.x[q], yv = sh.y[q], xl = PREC == 1 ? 0.0f : sh.xl[q], yl = PREC == 1 ? 0.0f : sh.yl[q];
          const float4* nh = nr.hi + p.off;
          const float2* nl = nr.lo + p.off;
          float run = 0.0f;
          int m = 0;
          for (int e = l; e < end.w; e += 32) {
            float4 h[4];
            float2 lo[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int ee = e + 8 * u;
              const int k2 = ee + (ee < end.x ? at.x : ee < end.y ? at.y : ee < end.z ? at.z : at.w);
              const bool in = ee < end.w;
              h[u] = in ? nh[k2] : make_float4(0.0f, 0.0f, 1.0f, 0.0f);
              lo[u] = in ? nl[k2] : make_float2(0.0f, 0.0f);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
              run += PREC == 1 ? near_term(h[u], lo[u], x, yv) : near_term(h[u], lo[u], x, yv, xl, yl, kw, &wide);
            if (++m == 8) { s += run; run = 0.0f; m = 0; }   // short runs: the sum stays accurate
          }
          s += run;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          s += __shfl_xor_sync(0xffffffffu, s, o);
          if (PREC == 0) wide += __shfl_xor_sync(0xffffffffu, wide, o);
        }
        if (l == 0) {
          sh.near[q] = s;
          if (PREC == 0) sh.wide[q] = wide;
        }
      }
      if (NW > 1) __syncthreads(); else __syncwarp();
      int a = 0;
      if (w == 0) {   // the decisions (mh_decide_f with the field's bound added to its guard)
        int open = 0;
        const Real cx = fx, cy = fy;
        if (ok) {
          if (ONE) far_part.eval(p, px, py);
          const float S = far_part.c0.x + sh.near[lane], b0 = far_part.c0.y + (PREC == 1 ? 0.0f : sh.wide[lane]);
          float dF, rn;
          const float Fn = near_field(p, ksc, S, fmaf(far_part.ty.y, 1.01f * fabsf(S), b0), &dF);
          const int take = near_decide(p, Fn, off ? INFINITY : dF, Fc, fe, rc, t0, t2, sh.lu[lane], &rn);
          open = take < 0;
          if (take == 1) {
            fx = ox; fy = oy; rc = rn; Fc = Fn; fe = dF;
            a = 1;
          }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, open);
        if (mask) { sh.cx[lane] = cx; sh.cy[lane] = cy; sh.ox[lane] = ox; sh.oy[lane] = oy; }
        if (lane == 0) sh.open = mask;
        if (ok && ((!ONE && a) || open)) {
          ax[k] = fx; ay[k] = fy; cs.fF[k] = Fc; cs.fsup[k] = rc; cs.fe[k] = fe;
        }
        if (ok && it < p.mh_jumps) {
          gx = sh.g[0][lane];
          gy = sh.g[1][lane];
          if (!ONE) { agx[k] = gx; agy[k] = gy; }
        }
      }
      if (NW > 1) __syncthreads(); else __syncwarp();
      const unsigned open = sh.open;
      for (unsigned o = open; o; o &= o - 1) {   // block-uniform
        const int q = __ffs(o) - 1;
        if constexpr (PREC == 1)
          a += near_open<NT>(p, pool, cs, wtab, plan_mh[d], kscale, tid == q, c, k, it, step, sh.ox[q], sh.oy[q],
                             sh.cx[q], sh.cy[q], sh.lu[q], &sh.ex);
        else
          a += near_open64<NT>(p, pool, cs, wtab, plan_mh[d], kscale, tid == q, c, k, it, step, sh.ox[q], sh.oy[q],
                               sh.cx[q], sh.cy[q], &sh.ex);
        if (ONE && tid == q) { fx = ax[k]; fy = ay[k]; Fc = cs.fF[k]; rc = cs.fsup[k]; fe = cs.fe[k]; }
      }
      if (w == 0) {
        const int acc = __popc(__ballot_sync(0xffffffffu, a)), rej = __popc(__ballot_sync(0xffffffffu, ok && !a));
        if (lane == 0 && !ONE && it > ndim_first)
          near_counts(p, y, nr.count + d, nr.progress + d, pr, plan[d].tiles, it, acc, rej);
        if (lane == 0 && ONE && it > ndim_first) {
          atomicAdd(nr.ring + 4 * d + (it & 3), (1ull << 44) | ((unsigned long long)acc << 22) | (unsigned long long)rej);
          if (it == p.mh_jumps && g == plan[d].item_off) {   // the step's last counts
            int A, R;
            if (!near_wait_counts(nr.ring + 4 * d + (it & 3), plan[d].tiles, &A, &R)) atomicAdd(gave_up, 1);
            else if (A + R > 0) y.MH_std = mh_std_clamp(p, std_ * mh_std_gain(A, R, &y.a_rate));
            else y.MH_std = std_;
          }
        }
        if (ONE && ok && it == p.mh_jumps) { ax[k] = fx; ay[k] = fy; cs.fe[k] = fe; }   // the last points (RD_MH_FINAL)
      }
    }
  }
}

// A lone diode's few items: eight warps each, the chains in registers (at most two
// blocks per SM; leaves larger diodes to k_mh_jumps_near).
template <int PREC>
__global__ void __launch_bounds__(256, 2)
k_mh_jumps_near_one(const DiodeParams* __restrict__ P, DiodeDyn* __restrict__ Dy, const __grid_constant__ Pool pool,
                    const PlanEntry* __restrict__ plan, const PlanHeader* __restrict__ ph,
                    const PlanEntry* __restrict__ plan_mh, const __grid_constant__ ChainState cs,
                    const int* __restrict__ ch_off, const double* __restrict__ wtab, const int* __restrict__ step_ptr,
                    int jumps, const __grid_constant__ NearState nr, double kscale, int* gave_up) {
  __shared__ NearShared<PREC, 8> sh;
  const int total = ph->total_items;
  if ((int)blockIdx.x >= total || total > (int)gridDim.x) return;
  near_jumps<PREC, 8, true>(sh, P, Dy, pool, plan, total, ph->n_diodes, plan_mh, cs, ch_off, wtab, *step_ptr, jumps, nr, kscale,
                      gave_up);
}

// Any number of items, four warps each; above: leaves plans of at most that many
// items to k_mh_jumps_near_one.
template <int PREC>
__global__ void __launch_bounds__(128, PREC == 1 ? 8 : 4)
k_mh_jumps_near(const DiodeParams* __restrict__ P, DiodeDyn* __restrict__ Dy, const __grid_constant__ Pool pool,
                const PlanEntry* __restrict__ plan, const PlanHeader* __restrict__ ph,
                const PlanEntry* __restrict__ plan_mh, const __grid_constant__ ChainState cs,
                const int* __restrict__ ch_off, const double* __restrict__ wtab, const int* __restrict__ step_ptr,
                int jumps, const __grid_constant__ NearState nr, double kscale, int* gave_up, int above) {
  __shared__ NearShared<PREC, 4> sh;
  const int total = ph->total_items;
  if ((int)blockIdx.x >= total || total <= above) return;
  near_jumps<PREC, 4, false>(sh, P, Dy, pool, plan, total, ph->n_diodes, plan_mh, cs, ch_off, wtab, *step_ptr, jumps, nr, kscale,
                       gave_up);
}
