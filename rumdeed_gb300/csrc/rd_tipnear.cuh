// rd_tipnear.cuh -- the jumps of the FP32 hyperboloid-tip Metropolis-Hastings chains
// from a near / far split of the field at the tip (included by rd_field.cu after
// rd_near.cuh, in its anonymous namespace).
//
// As on the planar cathode a jump only compares two targets, and the target depends on
// the point and the field F normal to the surface there, with log target = 2 log(-F) -
// rho (rho_entry_f's, less half the logarithm of the surface element's xi^2 - eta^2).
// F comes from an FP32 estimate with a rigorous bound on its distance from the pair
// sum's; near_decide answers where the bound allows only one answer, and a jump that it
// leaves open takes the pair sums of k_mh_jump_tip bit for bit (tip_open).  A last pass
// of that kernel (RD_MH_FINAL) gives the emission test the pair sums at the chains' last
// points.  So every chain is the one that the pair-sum jumps give.
//
// The surface is cut into panels (rings of equal arc length along the meridian, each
// into sectors about as wide; about RD_TN_PANELS), a panel with centre c and radius a.
// Electrons closer to c than 4 a are near: summed one by one, from a list of their
// offsets to c.  The others act through the expansion of their potential about c,
//   phi(x) = sum_n sum_m R_nm(x) conj(L_nm),  L_nm = sum_j S_nm(y_j),
//   R_nm = r^n P_nm e^(i m phi) / (n + m)!,  S_nm = (n - m)! P_nm e^(i m phi) / r^(n+1)
// (regular and irregular solid harmonics; Greengard and Rokhlin's local expansion), to
// degree RD_TN_DEG = 7, lengths in units of a.  Its gradient comes from
//   d/dz R_nm = R_(n-1)m,  (d/dx - i d/dy) R_nm = R_(n-1)(m-1),  (d/dx + i d/dy) R_nm = -R_(n-1)(m+1).
//
// The bound.  The degree-n part of a unit charge's field at distance <= a from c is at
// most n t^(n-1) / D^2, t = a / D, so the parts left out add up to at most
//   sum_far sum_(n>7) n t^(n-1) / D^2 <= sum_far 8 t^7 / (D - a)^2.
// Roundings are multiples of u = 2^-24 times the sum of the terms' magnitudes B =
// sum_near 1 / d^2 + sum_far 1 / (D - a)^2: the pair sum's tiles of 128 terms one after
// another (132 u with the tiles' two-sums) and its terms (28 u: the difference, the
// reciprocal root's 2 ulp three times, the products); here a near term's 28 u, 40 u and
// the list's length / 256 of its sum, 20 u for the normal; and for a far electron its
// coefficients' recurrences (60 u) and their sum over the electrons.  A near electron's
// offset and the point's are rounded to u a few times a: 16 u a times the gradient's
// 2 / d^3.  The sphere's image charges enter scaled by K = q0 / (4 pi eps0) ~ 1e-9; an
// electron outside the sphere has its image term bounded by K (1 + dis / R) / d^2, so
// they only widen the bound.  A panel that sees an electron inside the sphere, a charge
// that is not an electron's or a full list leaves all its jumps open.
#pragma once

#define RD_TN_DEG 7
#define RD_TN_NEAR 4.0f       // near electrons: closer to the panel's centre than this many radii

// Does the diode's step run its jumps here?  (planner mode PM_MH_TIP)
__device__ __forceinline__ bool tip_live(const DiodeParams& p, const DiodeDyn& y) {
  return p.active && p.emission && p.tn && y.chains > 0;
}

// Lists and expansions of every panel, one panel per block and turn.  Bound by the
// recurrences of the far electrons (about 230 FP32 instructions each): 12,500 electrons
// take 83 us with 512 panels, 226 us with 1536.  Fewer panels have longer lists; a step of
// 5000 electrons close to the tip and 14,000 chains takes 4.7 / 4.2 / 4.0 ms with 256 / 512
// / 768 panels, one of 9000 spread electrons and 12,100 chains 3.9 / 3.6 / 3.6 ms.
__global__ void __launch_bounds__(256)
k_tip_panels(const DiodeParams* __restrict__ P, const DiodeDyn* __restrict__ Dy, Pool pool, NearState nr, int per) {
  constexpr int D = RD_TN_DEG;
  __shared__ float red[8][68];
  __shared__ int s_n, s_at, s_bad;
  const int d = blockIdx.x / per, b = blockIdx.x % per, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const DiodeParams& p = P[d];
  if (!tip_live(p, Dy[d])) return;
  const int n = Dy[d].n;
  if (b == 0 && tid == 0) near_reset(p, nr, d, Dy[d].MH_std);
  const float4* hi = pool.pk_hi + p.off;
  const float4* lo = pool.pk_lo + p.off;
  const float R = (float)(p.r_tip * 1.0e9), z0 = (float)((p.h_tip - p.r_tip) * 1.0e9);
  for (int k = b; k < p.tn_np; k += per) {
    const float4 c = p.tn_pan[k];
    const float near2 = (RD_TN_NEAR * c.w) * (RD_TN_NEAR * c.w), ia = 1.0f / c.w;
    // the near electrons' number, a place for their list, and whether the bound holds
    int cnt = 0, bad = 0;
    for (int j = tid; j < n; j += 256) {
      const float4 h = hi[j], l = lo[j];
      const float x = (h.x - c.x) + l.x, y = (h.y - c.y) + l.y, z = (h.z - c.z) + l.z;
      cnt += fmaf(z, z, fmaf(y, y, x * x)) < near2;
      const float zs = h.z - z0;
      bad |= !(fmaf(zs, zs, fmaf(h.y, h.y, h.x * h.x)) > 0.999f * R * R && h.w == -1.0f);
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (tid == 0) { s_n = 0; s_bad = 0; }
    __syncthreads();
    if (lane == 0 && cnt) atomicAdd(&s_n, cnt);
    if (bad) s_bad = 1;
    __syncthreads();
    cnt = s_n;
    if (tid == 0) {
      s_at = __ldcg(p.tn_next) <= p.tn_cap ? atomicAdd(p.tn_next, cnt) : -1;
      if (s_at < 0 || (long long)s_at + cnt > p.tn_cap) s_bad = 1;
    }
    __syncthreads();
    bad = s_bad;
    const int at = s_at;
    __syncthreads();
    if (tid == 0) s_n = 0;
    __syncthreads();
    if (!bad) {   // block-uniform
      float cr[D + 1][D + 1], ci[D + 1][D + 1];   // sums of S_nm
#pragma unroll
      for (int m = 0; m <= D; ++m)
#pragma unroll
        for (int q = 0; q <= D; ++q) cr[m][q] = ci[m][q] = 0.0f;
      float T = 0.0f, B = 0.0f;
      for (int j0 = 0; j0 < n; j0 += 256) {
        const int j = j0 + tid;
        float x = 0.0f, y = 0.0f, z = 0.0f;
        int in = 0;
        if (j < n) {
          const float4 h = hi[j], l = lo[j];
          x = (h.x - c.x) + l.x; y = (h.y - c.y) + l.y; z = (h.z - c.z) + l.z;
          in = fmaf(z, z, fmaf(y, y, x * x)) < near2 ? 1 : 2;
        }
        const unsigned m1 = __ballot_sync(0xffffffffu, in == 1);
        if (m1) {
          int b = 0;
          if (lane == 0) b = atomicAdd(&s_n, __popc(m1));
          b = __shfl_sync(0xffffffffu, b, 0);
          b += __popc(m1 & ((1u << lane) - 1));
          if (in == 1 && b < cnt) p.tn_list[(size_t)at + b] = make_float4(x, y, z, 0.0f);
        }
        if (in == 2) {
          x *= ia; y *= ia; z *= ia;
          const float r2 = fmaf(z, z, fmaf(y, y, x * x)), inv = rsqrtf(r2), i2 = inv * inv;
          const float xi = x * i2, yi = y * i2, zi = z * i2, q = 1.0f / (r2 * inv - 1.0f), q2 = q * q;
          const float t3 = (inv * inv) * inv;
          B += q2;
          T = fmaf((t3 * t3) * inv, q2, T);
          float mr = inv, mi = 0.0f;   // S_mm
#pragma unroll
          for (int m = 0; m <= D; ++m) {
            if (m > 0) {
              const float f = (float)(2 * m - 1), tr = f * (mr * xi - mi * yi), ti = f * (mr * yi + mi * xi);
              mr = tr; mi = ti;
            }
            float ar = mr, ai = mi, br = 0.0f, bi = 0.0f;   // S_nm and the one before it
#pragma unroll
            for (int q1 = m; q1 <= D; ++q1) {
              if (q1 > 0) { cr[m][q1] += ar; if (m > 0) ci[m][q1] += ai; }
              if (q1 < D) {
                const float f = (float)(2 * q1 + 1) * zi, g = (float)(q1 * q1 - m * m) * i2;
                const float tr = fmaf(f, ar, -(g * br)), ti = fmaf(f, ai, -(g * bi));
                br = ar; bi = ai; ar = tr; ai = ti;
              }
            }
          }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        B += __shfl_xor_sync(0xffffffffu, B, o);
        T += __shfl_xor_sync(0xffffffffu, T, o);
      }
      if (lane == 0) { red[w][64] = B; red[w][65] = T; }
      int at_v = 0;
#pragma unroll
      for (int m = 0; m <= D; ++m)
#pragma unroll
        for (int q = m > 0 ? m : 1; q <= D; ++q)
#pragma unroll
          for (int part = 0; part < (m > 0 ? 2 : 1); ++part) {
            float v = part ? ci[m][q] : cr[m][q];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) red[w][at_v] = v;
            ++at_v;
          }
      __syncthreads();
      if (tid < 64) {   // L_qm at [m][q]; zero where q < m or q = 0
        const int m = tid >> 3, q = tid & 7;
        float2 v = make_float2(0.0f, 0.0f);
        if (q > 0 && q >= m) {
          int idx = m == 0 ? q - 1 : D;   // D of m = 0, then pairs
          for (int mm = 1; mm < m; ++mm) idx += 2 * (D + 1 - mm);
          if (m > 0) idx += 2 * (q - m);
          for (int ww = 0; ww < 8; ++ww) {
            v.x += red[ww][idx];
            if (m > 0) v.y += red[ww][idx + 1];
          }
        }
        p.tn_rec[(size_t)k * 64 + tid] = v;
      }
      if (tid == 64) {
        float Bs = 0.0f, Ts = 0.0f;
        for (int ww = 0; ww < 8; ++ww) { Bs += red[ww][64]; Ts += red[ww][65]; }
        const float u = 5.97e-8f, ia2 = 1.02f * ia * ia;
        // (what the expansion may be off; the magnitudes; the list)
        p.tn_hdr[k] = make_float4(ia2 * fmaf(8.0f, Ts, (60.0f + 8.0f + (float)((n + 255) / 256 + 5)) * u * Bs), ia2 * Bs,
                                  __int_as_float(at), __int_as_float(cnt));
      }
    } else if (tid == 0) {
      p.tn_hdr[k] = make_float4(INFINITY, 0.0f, __int_as_float(0), __int_as_float(0));
    }
    __syncthreads();
  }
}

// The entry (t0, t2) of rho_entry_f at a tip point.
__device__ __forceinline__ void tip_entry(const DiodeParams& p, double xi, float* t0, float* t2) {
  *t0 = tip_log_phi(p, (float)(xi * xi - p.eta_1 * p.eta_1));
  *t2 = p.tn_t2;
}

// A jump that the estimate leaves open (rare): the pair sums at the proposal (point 0)
// and at the chain's point (1), as k_mh_jump_tip forms them, by the whole block -- a
// thread per tile and point's 128 terms, then each component's tiles in order -- and its
// test.  FP64 latency on few threads, so log u is drawn by another warp meanwhile; with
// one thread for both points of a tile and log u at the end a step with eight open jumps
// took 3.23 ms, so 3.15.  A chain that has not moved keeps the field of its start.  mine decides.
template <int NT>
struct TipExact {
  float t[2][6][NT / 2];        // a pass's tile sums
  float4 ih[2], iih[2];
  double X[2], Y[2], Z[2], f[2][3], F[2], s[2], lu;
};
template <int NT>
__device__ __noinline__ int tip_open(const DiodeParams& p, const Pool& pool, const ChainState& cs, const PlanEntry& e,
                                     double kscale, bool mine, int c, int k, int it_idx, uint32_t step, double nxi,
                                     double nph, double cxi, double cph, TipExact<NT>* s) {
  const int tid = threadIdx.x, n = e.n_j, tiles = (n + RD_TILE - 1) / RD_TILE, tpc = e.clen / RD_TILE;
  if (tid < 2) {
    double X, Y, Z;
    tip_grid_xyz(p, tid ? cxi : nxi, tid ? cph : nph, &X, &Y, &Z);
    float4 il, iil;
    point_pack(p, X, Y, Z, s->ih[tid], il, s->iih[tid], iil);
    s->X[tid] = X; s->Y[tid] = Y; s->Z[tid] = Z;
  } else if (tid == 32) {   // log u of the accept test
    double u1, u2;
    rng2(p.seed, (uint32_t)c, (uint32_t)it_idx, step, RNG_ACCEPT, &u1, &u2);
    s->lu = log(u1);
  }
  __syncthreads();
  const int pt = tid / 3, i = tid % 3;   // threads 0..5: component i of point pt
  float h = 0.0f, l = 0.0f, im = 0.0f;
  double acc = 0.0;
  int in_chunk = 0, chunk = 0;
  for (int base = 0; base < tiles; base += NT / 2) {
    const int q = tid / (NT / 2), slot = tid % (NT / 2), tile = base + slot;   // a thread per point and tile
    if (tile < tiles) {
      const int j = tile * RD_TILE;
      const float4 ih[1] = {s->ih[q]}, iih[1] = {s->iih[q]};
      float td[1][3] = {{0.f, 0.f, 0.f}}, te[1][3] = {{0.f, 0.f, 0.f}};
      const float4 *sh = pool.pk_hi + p.off + j, *sl = pool.pk_lo + p.off + j;
      const int kmax = min(RD_TILE, n - j);
      if (p.image_charge) tip_point_tiles_f32<1, false, true>(sh, sl, kmax, ih, iih, td, te);
      else tip_point_tiles_f32<1, false, false>(sh, sl, kmax, ih, iih, td, te);
      for (int a = 0; a < 3; ++a) { s->t[q][a][slot] = td[0][a]; s->t[q][3 + a][slot] = te[0][a]; }
    }
    __syncthreads();
    if (tid < 6)
      for (int t = 0; t < min(NT / 2, tiles - base); ++t) {
        two_sum_acc(h, l, s->t[pt][i][t]);
        im += s->t[pt][3 + i][t];
        if (++in_chunk == tpc || base + t + 1 == tiles) {
          const double f = tip_sum_finish(p, h, l, im, s->iih[pt].w, kscale);
          acc = chunk == 0 ? f : acc + f;
          ++chunk;
          h = l = im = 0.0f;
          in_chunk = 0;
        }
      }
    __syncthreads();
  }
  if (tid < 6) s->f[pt][i] = acc;
  __syncthreads();
  if (tid < 2) {
    const double f3[3] = {s->f[tid][0], s->f[tid][1], s->f[tid][2]};
    s->F[tid] = tip_normal_field(p, s->X[tid], s->Y[tid], s->Z[tid], f3);
    s->s[tid] = s->F[tid] < 0.0 ? tip_target_log(p, s->F[tid], tid ? cxi : nxi) : 0.0;
  }
  __syncthreads();
  int a = 0;
  if (mine) {
    float t0, t2;
    const double F = s->F[0], Fc = cs.em[k] ? s->F[1] : cs.F[k], sn = s->s[0], sc = cs.em[k] ? s->s[1] : cs.sup[k];
    if (F < 0.0) {
      a = sn >= sc || s->lu <= sn - sc;
    }
    const double xi = a ? nxi : cxi;
    const float Ff = (float)(a ? F : Fc);
    tip_entry(p, xi, &t0, &t2);
    cs.fF[k] = Ff;
    cs.fe[k] = 1.2e-7f * fabsf(Ff);
    cs.fsup[k] = rho_entry_f(p, t0, t2, Ff);
    if (a) { cs.x[k] = nxi; cs.y[k] = nph; cs.em[k] = 1; }
  }
  __syncthreads();
  return a;
}

struct TipShared {
  float4 r[32];                     // proposal: offset to the panel's centre (nm), radius of the panel
  int pan[32];                      // its panel; -1: no chain
  float f[32][3], B[32], C[32], lu[32];
  double g[2][32];                  // next Gaussian pair
  double oxi[32], oph[32], cxi[32], cph[32];
  float rc[7][8];                   // 1 / ((n + 1)^2 - m^2) at [m][n]
  unsigned open;
  int dead;
  TipExact<256> ex;
};

// Every jump of every chain of those diodes, in one cooperative launch; the structure is
// k_mh_jumps_near's: 32 chains per item, a diode's progress word between its jumps
// (waits bounded by RD_NEAR_SPIN polls).  Warp 0 proposes (FP64, as k_mh_propose) and
// decides; eight lanes per chain sum its near electrons, four loads in flight each, and
// evaluate the expansion, an order m per lane.  em marks a chain that has moved.
// Measured (GB300, 8900 chains, 12,500 electrons, 80 jumps): 17.1 ms with the pair-sum
// jumps, 1.7 ms so, the panels and the last pass included.  Bound by the latency of a
// jump, about 10 us: FP64 sine and cosine 3, the step 1.5, the sums 3, the decision 1.4,
// the rest loads and the progress word.  One jump in 10^5 is left open (tip_open);
// the estimate lies within 0.11 of its bound at the chains' last points (tests/near_bound.cu).
__global__ void __launch_bounds__(256, 2)
k_tip_jumps(const DiodeParams* __restrict__ P, DiodeDyn* __restrict__ Dy, const __grid_constant__ Pool pool,
            const PlanEntry* __restrict__ plan, const PlanHeader* __restrict__ ph, const PlanEntry* __restrict__ plan_mh,
            const __grid_constant__ ChainState cs, const int* __restrict__ ch_off, const int* __restrict__ step_ptr,
            int jumps, const __grid_constant__ NearState nr, double kscale, int* gave_up) {
  __shared__ TipShared sh;
  const int total = ph->total_items, nd = ph->n_diodes, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if ((int)blockIdx.x >= total) return;
  if (tid == 0) sh.dead = 0;
  if (tid < 56) {
    const int m = tid >> 3, q = tid & 7;
    sh.rc[m][q] = q >= m ? 1.0f / (float)((q + 1) * (q + 1) - m * m) : 0.0f;
  }
  __syncthreads();
  const double twopi = 2.0 * c_k.pi;
  const float ksc = (float)kscale;
  for (int it = 1; it <= jumps; ++it) {
    for (int g = blockIdx.x; g < total; g += gridDim.x) {
      const int d = near_entry(plan, nd, g, lane);
      const DiodeParams& p = P[d];
      if (it > p.mh_jumps) continue;
      DiodeDyn& y = Dy[d];
      const int ndim_first = (int)nint_d(p.mh_jumps * 0.25);
      const int M = plan[d].n_i, c = (g - plan[d].item_off) * 32 + lane, k = ch_off[d] + c;
      const uint32_t step = (uint32_t)(*step_ptr - y.step_offset);
      float t0 = 0.0f, t2 = 0.0f, Fv = 0.0f, nx = 0.0f, ny = 0.0f, nz = 0.0f, ev = 0.0f, wide = 0.0f;
      double nxi = 1.0, nph = 0.0, cxi = 1.0, cph = 0.0;
      int ok = 0, inside = 0, pan = -1;
      unsigned long long pr = 0;
      if (w == 7 && c < M && it < p.mh_jumps && cs.ok[k]) {   // the next proposal's Gaussian pair
        double g1, g2;
        gauss2(p.seed, (uint32_t)c, (uint32_t)(it + 1), step, &g1, &g2);
        sh.g[0][lane] = g1;
        sh.g[1][lane] = g2;
      }
      if (w == 1 && c < M) {   // log u of the accept test
        uint32_t o[4];
        philox4x32((uint32_t)c, (uint32_t)it, step, RNG_ACCEPT, (uint32_t)p.seed, (uint32_t)(p.seed >> 32), o);
        sh.lu[lane] = logf(fmaf((float)(o[1] >> 11), 1.1102230246251565e-16f, (float)o[0] * 2.3283064365386963e-10f));
      }
      if (w == 0) {
        ok = c < M ? cs.ok[k] : 0;
        double g1 = 0.0, g2 = 0.0;
        if (ok) {
          cxi = cs.x[k]; cph = cs.y[k];
          if (it == 1) gauss2(p.seed, (uint32_t)c, 1u, step, &g1, &g2);
          else { g1 = cs.gx[k]; g2 = cs.gy[k]; }
        }
        if (lane == 0) {   // the step size after the last jump
          const volatile unsigned long long* prog = nr.progress + d;
          pr = *prog;
          const int need = it - 1 > ndim_first ? it - 1 : 0;   // the warm-up's step size is fixed: no wait
          for (int spins = 0; (int)((unsigned)pr & ~RD_NEAR_CLAMPED) < need && spins < RD_NEAR_SPIN; ++spins) pr = *prog;
          if ((int)((unsigned)pr & ~RD_NEAR_CLAMPED) < need) sh.dead = 1;
        }
        pr = __shfl_sync(0xffffffffu, pr, 0);
        __threadfence();   // MH_std was written before the progress word
        const double mhs = __ldcg(&y.MH_std);
        float4 r = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        if (ok) {   // the proposal of k_mh_propose
          const double sxi = (it > ndim_first) ? (p.max_xi - 1.0) * mhs : (p.max_xi - 1.0) * 0.10;
          const double sph = (it > ndim_first) ? twopi * mhs : twopi * 0.10;
          inside = tip_step(p, cxi, cph, g1, g2, sxi, sph, &nxi, &nph);
        }
        if (inside) {
          double X, Y, Z;
          tip_xyz(p, nxi, p.eta_1, nph, &X, &Y, &Z);
          X *= 1.0e9; Y *= 1.0e9; Z *= 1.0e9;
          const float px = (float)X, py = (float)Y, pz = (float)Z;   // tip_grid_xyz's point
          const float ox = (float)((double)px - X), oy = (float)((double)py - Y), oz = (float)((double)pz - Z);
          const int2 ring = p.tn_map[min((int)(sqrtf((float)(nxi - 1.0)) * p.tn_vs), RD_TN_MAP - 1)];
          const int sec = (int)((float)nph * 0.15915494f * (float)ring.y);
          pan = ring.x + max(min(sec, ring.y - 1), 0);
          const float4 ct = p.tn_pan[pan];
          r = make_float4(px - ct.x, py - ct.y, pz - ct.z, ct.w);
          const float v = (float)(nxi * nxi - p.eta_1 * p.eta_1), iv = 1.0f / v;
          t0 = tip_log_phi(p, v);
          t2 = p.tn_t2;
          // the normal
          const float rho2 = fmaf(px, px, py * py), gn = p.tn_nf * rsqrtf(rho2 + p.tn_c);
          nz = rsqrtf(fmaf(gn * gn, rho2, 1.0f));
          nx = -(gn * px) * nz;
          ny = -(gn * py) * nz;
          // vacuum field: normal to the surface, |E| = pre_E / sqrt((xi^2 - eta^2)(1 - eta^2)), to
          // first order at a point off the surface by the FP32 grid (ox, oy, oz): d eta along the
          // normal, d xi along the meridian
          const float es = (float)p.eta_1, g2 = p.tn_e2, ihe = sqrtf(g2 * iv) * p.tn_ia;
          const float de = fmaf(nx, ox, fmaf(ny, oy, nz * oz)) * ihe, ir = rsqrtf(fmaxf(rho2, 1.0e-12f));
          const float orho = fmaf(px, ox, py * oy) * ir, xf = (float)nxi;
          const float dx = fmaf(nz, orho, gn * (rho2 * ir) * nz * oz) * sqrtf(fmaf(xf, xf, -1.0f) * iv) * p.tn_ia;
          Fv = p.tn_v0 * rsqrtf(v);
          Fv = fmaf(Fv, fmaf(fmaf(es, iv, es / g2), de, -(xf * iv) * dx), Fv);
          const float big = fmaxf(fmaxf(fabsf(px), fabsf(py)), fabsf(pz));
          ev = fabsf(Fv) * (8.0e-7f + 1.0e-8f * big * p.tn_ir);
          // image charges: K (1 + dis / R) with some room
          const float zs = pz - p.tn_z0;
          wide = p.image_charge ? 3.0e-9f * (1.0f + sqrtf(fmaf(zs, zs, rho2)) * p.tn_ir) : 0.0f;
          // tip_field_E drops the lateral field where xi - 1 < 1e-6: 2 (xi - 1) eta^2 / (1 - eta^2) of F
          if (nxi - 1.0 < 1.3e-6) ev = fmaf(fabsf(Fv), 3.0e-6f * p.tn_nf * p.tn_nf, ev);
          if (!(fmaf(r.z, r.z, fmaf(r.y, r.y, r.x * r.x)) <= r.w * r.w)) ev = INFINITY;
        }
        sh.r[lane] = r;
        sh.pan[lane] = pan;
      }
      __syncthreads();
      if (sh.dead) {   // block-uniform
        if (tid == 0) atomicAdd(gave_up, 1);
        return;
      }
      {   // the field's sums, eight lanes per chain
        const int l = lane & 7, q = w * 4 + (lane >> 3), pn = sh.pan[q];
        float sx = 0.0f, sy = 0.0f, sz = 0.0f, B = 0.0f, C = 0.0f;
        if (pn >= 0) {
          const float4 pt = sh.r[q], hd = p.tn_hdr[pn];
          const float2* rec = p.tn_rec + (size_t)pn * 64;
          // columns m - 1, m, m + 1 of the coefficients, n = 0..7 (lane 7: none)
          float4 c0[4], c1[4], c2[4];
          const bool far = l < RD_TN_DEG;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            c0[u] = far && l > 0 ? reinterpret_cast<const float4*>(rec + 8 * (l - 1))[u] : zero;
            c1[u] = far ? reinterpret_cast<const float4*>(rec + 8 * l)[u] : zero;
            c2[u] = far ? reinterpret_cast<const float4*>(rec + 8 * (l + 1))[u] : zero;
          }
          const float4* list = p.tn_list + __float_as_int(hd.z);
          const int cnt = __float_as_int(hd.w);
          float rx = 0.0f, ry = 0.0f, rz = 0.0f;
          int m8 = 0;
          for (int e = l; e < cnt; e += 32) {
            float4 h[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) h[u] = e + 8 * u < cnt ? list[e + 8 * u] : make_float4(1.0e18f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const float dx = pt.x - h[u].x, dy = pt.y - h[u].y, dz = pt.z - h[u].z;
              const float inv = rsqrtf(fmaf(dz, dz, fmaf(dx, dx, fmaf(dy, dy, 1e-20f)))), i2 = inv * inv, i3 = i2 * inv;
              rx = fmaf(i3, dx, rx); ry = fmaf(i3, dy, ry); rz = fmaf(i3, dz, rz);
              B += i2;
              C += i3;
            }
            if (++m8 == 8) { sx -= rx; sy -= ry; sz -= rz; rx = ry = rz = 0.0f; m8 = 0; }
          }
          sx -= rx; sy -= ry; sz -= rz;
          if (far) {   // the expansion's orders m = l
            const float ia = 1.0f / pt.w, a = pt.x * ia, b = pt.y * ia, z = pt.z * ia;
            const float r2 = fmaf(z, z, fmaf(b, b, a * a));
            float Rr = 1.0f, Ri = 0.0f, br = 0.0f, bi = 0.0f, gx = 0.0f, gy = 0.0f, gz = 0.0f;
#pragma unroll
            for (int m = 1; m < RD_TN_DEG; ++m)
              if (m <= l) {
                const float f = 0.5f / (float)m, tr = f * (Rr * a - Ri * b), ti = f * (Rr * b + Ri * a);
                Rr = tr; Ri = ti;
              }
            const float wz = l == 0 ? 1.0f : 2.0f;
#pragma unroll
            for (int n1 = 0; n1 < RD_TN_DEG; ++n1)
              if (n1 >= l) {
                const int nn = n1 + 1;
                auto at = [nn](const float4* cc) {
                  const float4 v4 = cc[nn >> 1];
                  return (nn & 1) ? make_float2(v4.z, v4.w) : make_float2(v4.x, v4.y);
                };
                const float2 Lm = at(c0), Lz = at(c1), Lp = at(c2);
                // conj(L) R
                gz = fmaf(wz, fmaf(Lz.x, Rr, Lz.y * Ri), gz);
                gx += fmaf(Lp.x, Rr, Lp.y * Ri) - fmaf(Lm.x, Rr, Lm.y * Ri);
                gy -= fmaf(Lp.x, Ri, -(Lp.y * Rr)) + fmaf(Lm.x, Ri, -(Lm.y * Rr));
                const float f = (float)(2 * n1 + 1) * z, rc = sh.rc[l][n1];
                const float tr = fmaf(f, Rr, -(r2 * br)) * rc, ti = fmaf(f, Ri, -(r2 * bi)) * rc;
                br = Rr; bi = Ri; Rr = tr; Ri = ti;
              }
            const float ia2 = ia * ia;
            sx = fmaf(gx, ia2, sx); sy = fmaf(gy, ia2, sy); sz = fmaf(gz, ia2, sz);
          }
#pragma unroll
          for (int o = 4; o > 0; o >>= 1) {
            const unsigned grp = 0xffu << (lane & 24);
            sx += __shfl_xor_sync(grp, sx, o); sy += __shfl_xor_sync(grp, sy, o); sz += __shfl_xor_sync(grp, sz, o);
            B += __shfl_xor_sync(grp, B, o); C += __shfl_xor_sync(grp, C, o);
          }
          if (l == 0) {   // the sums and the bound on them
            const float u = 5.97e-8f;
            sh.f[q][0] = sx; sh.f[q][1] = sy; sh.f[q][2] = sz;
            sh.B[q] = 1.01f * B + hd.y;
            sh.C[q] = hd.x + u * ((250.0f + (float)(cnt >> 8)) * (1.01f * B) + 200.0f * hd.y + 34.0f * pt.w * (1.01f * C));
          }
        }
      }
      __syncthreads();
      int a = 0;
      if (w == 0) {
        int open = 0;
        if (inside) {
          const float S = fmaf(nx, sh.f[lane][0], fmaf(ny, sh.f[lane][1], nz * sh.f[lane][2]));
          const float Fn = fmaf(ksc, S, Fv);
          const float dF = fmaf(ksc, fmaf(wide, sh.B[lane], sh.C[lane]), ev) + 8.0e-7f * (fabsf(Fv) + fabsf(ksc * S));
          float rn;
          const int take = near_decide(p, Fn, dF, cs.fF[k], cs.fe[k], cs.fsup[k], t0, t2, sh.lu[lane], &rn);
          open = take < 0;
          if (take == 1) {
            cs.x[k] = nxi; cs.y[k] = nph; cs.fF[k] = Fn; cs.fe[k] = dF; cs.fsup[k] = rn; cs.em[k] = 1;
            a = 1;
          }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, open);
        if (open) { sh.oxi[lane] = nxi; sh.oph[lane] = nph; sh.cxi[lane] = cxi; sh.cph[lane] = cph; }
        if (lane == 0) sh.open = mask;
        if (ok && it < p.mh_jumps) { cs.gx[k] = sh.g[0][lane]; cs.gy[k] = sh.g[1][lane]; }
      }
      __syncthreads();
      for (unsigned o = sh.open; o; o &= o - 1) {   // block-uniform
        const int q = __ffs(o) - 1;
        a += tip_open<256>(p, pool, cs, plan_mh[d], kscale, tid == q, c - lane + q, k, it, step, sh.oxi[q], sh.oph[q], sh.cxi[q],
                           sh.cph[q], &sh.ex);
      }
      if (w == 0) {
        const int acc = __popc(__ballot_sync(0xffffffffu, a)), rej = __popc(__ballot_sync(0xffffffffu, ok && !a));
        if (lane == 0 && it > ndim_first) near_counts(p, y, nr.count + d, nr.progress + d, pr, plan[d].tiles, it, acc, rej);
      }
      __syncthreads();   // the shared proposals are free for the next item
    }
  }
}
