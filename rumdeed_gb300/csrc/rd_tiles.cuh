// rd_tiles.cuh -- per-pair arithmetic of one shared-memory j-tile, shared by
// the force kernels (i = particle) and the field kernels (i = evaluation
// point, always in the upper role: the point images / is imaged as the "a"
// argument of the reference image functions).
#pragma once
#include "rd_f64.cuh"
#include "rd_pair.cuh"

enum { T_UPPER = 0, T_LOWER = 1, T_DIAG = 2 };

struct F32Acc {
  float hx, lx, hy, ly, hz, lz;
  __device__ void zero() { hx = lx = hy = ly = hz = lz = 0.f; }
  __device__ void add(float tx, float ty, float tz) {
    two_sum_acc(hx, lx, tx);
    two_sum_acc(hy, ly, ty);
    two_sum_acc(hz, lz, tz);
  }
};

// ---- planar, FP32 compensated ------------------------------------------------
// One j-tile against the thread's particle i.  NIC0: N_ic_max == 0 fast path.
// ELEC (tiles whose charges are all -1, the electrons' q/q0; not the
// diagonal tile): the charge is a constant, so its multiplies fold into signs.
template <int MODE, bool NIC0, bool ELEC = false>
__device__ __forceinline__ void planar_tile_f32(const float4* __restrict__ sh, const float4* __restrict__ sl,
                                                int kmax, float4 ih, float4 il, int self_k,
                                                int nic, float dnm, int ic, float& tx,
                                                float& ty, float& tz) {
  float sx = 0.f, sy = 0.f, sz = 0.f, szs = 0.f;
#pragma unroll 4
  for (int k = 0; k < kmax; ++k) {
    float4 h = sh[k], l = sl[k];
    float q = ELEC ? -1.f : h.w;
    if (MODE == T_DIAG) q = (k == self_k) ? 0.f : q;
    float dx = (ih.x - h.x) + (il.x - l.x);
    float dy = (ih.y - h.y) + (il.y - l.y);
    float dz = (ih.z - h.z) + (il.z - l.z);
    float dxy2 = fmaf(dx, dx, dy * dy);
    float r2 = fmaf(dz, dz, dxy2);
    float inv = rsqrtf(fmaxf(r2, 1e-20f));
    float s = q * (inv * inv) * inv;
    sx = fmaf(s, dx, sx);
    sy = fmaf(s, dy, sy);
    sz = fmaf(s, dz, sz);
    if (ic) {
      // n = 0 partner at -z_b: dz = z_a + z_b (symmetric in the roles)
      float zs = (ih.z + h.z) + (il.z + l.z);
      float ri = rsqrtf(fmaxf(fmaf(zs, zs, dxy2), 1e-20f));
      float si = q * (ri * ri) * ri;
      sx = fmaf(-si, dx, sx);
      sy = fmaf(-si, dy, sy);
      sz = fmaf(-si, zs, sz);
      if (!NIC0) {
        // anode distances u = d - z, exact near the anode
        float us = il.w + l.w;
        for (int n = 1; n <= nic; ++n) {
          float two_nd = 2.0f * n * dnm;
          // opposite-charge partners (symmetric in the roles)
          float z1 = (n == 1) ? -us : zs - two_nd;   // z_a + z_b - 2nd
          float z2 = zs + two_nd;                      // z_a + z_b + 2nd
          float r1 = rsqrtf(fmaxf(fmaf(z1, z1, dxy2), 1e-20f));
          float r2b = rsqrtf(fmaxf(fmaf(z2, z2, dxy2), 1e-20f));
          float s1 = q * (r1 * r1) * r1, s2 = q * (r2b * r2b) * r2b;
          sx = fmaf(-(s1 + s2), dx, sx);
          sy = fmaf(-(s1 + s2), dy, sy);
          sz = fmaf(-s1, z1, fmaf(-s2, z2, sz));
          // same-charge partners, evaluated with a = i; the z part changes
          // sign when j < i (lower-index role convention)
          float z3 = dz - two_nd, z4 = dz + two_nd;
          float r3 = rsqrtf(fmaxf(fmaf(z3, z3, dxy2), 1e-20f));
          float r4 = rsqrtf(fmaxf(fmaf(z4, z4, dxy2), 1e-20f));
          float s3 = q * (r3 * r3) * r3, s4 = q * (r4 * r4) * r4;
          sx = fmaf(s3 + s4, dx, sx);
          sy = fmaf(s3 + s4, dy, sy);
          float zsame = fmaf(s3, z3, s4 * z4);
          if (MODE == T_DIAG) zsame = (k > self_k) ? zsame : -zsame;
          szs += zsame;
        }
      }
    }
  }
  if (!NIC0) {
    if (MODE == T_LOWER) szs = -szs;
    sz += szs;
  }
  tx += sx; ty += sy; tz += sz;
}

// ---- planar, FP64 --------------------------------------------------------------
// One pair (i, j) of acc_ic_planar_series.inc's sum, without the factor q_i k: the
// Coulomb term plus, with image charges on, the partners' with i in the "a" role
// when upper and j in it otherwise (the x, y parts then change sign: force_ic_N).
// Every term shares dx, dy, so their inverse cubes are added up first.  25 FP64
// operations with one image partner (50 with sqrt and division, rd_f64.cuh).
__device__ __forceinline__ double planar_inv_f64(double s, double L2, float L2x3) {
  return rd_cube_ok(s) ? rd_inv_cube(s, L2x3) : rd_inv_cube_any(s, L2);
}
__device__ __forceinline__ void planar_pair_f64(const rd_d4& pj, double x1, double y1, double z1, bool upper, int nic,
                                                double d, int ic, double L2, float L2x3, double& ax, double& ay,
                                                double& az) {
  const double dx = x1 - pj.x, dy = y1 - pj.y, dz = z1 - pj.z;
  const double dxy2 = fma(dx, dx, dy * dy);
  const double r2 = fma(dz, dz, dxy2);
  double t, tz;
  if (ic) {
    const double zs = z1 + pj.z, s2 = fma(zs, zs, dxy2);   // the n = 0 partner at -z
    double inv, ini;
    if (rd_cube_ok(r2) && rd_cube_ok(s2)) {
      inv = rd_inv_cube(r2, L2x3);
      ini = rd_inv_cube(s2, L2x3);
    } else {
      inv = rd_inv_cube_any(r2, L2);
      ini = rd_inv_cube_any(s2, L2);
    }
    t = inv - ini;
    tz = fma(inv, dz, -(ini * zs));
    const double da = upper ? dz : -dz;
    for (int n = 1; n <= nic; ++n) {
      const double nd = (2.0 * n) * d;
      const double h0 = zs - nd, h1 = zs + nd, h2 = da - nd, h3 = da + nd;   // partners at 2nd - z, -2nd - z, 2nd + z, -2nd + z
      const double i0 = planar_inv_f64(fma(h0, h0, dxy2), L2, L2x3), i1 = planar_inv_f64(fma(h1, h1, dxy2), L2, L2x3);
      const double i2 = planar_inv_f64(fma(h2, h2, dxy2), L2, L2x3), i3 = planar_inv_f64(fma(h3, h3, dxy2), L2, L2x3);
      t += (i2 + i3) - (i0 + i1);
      tz = fma(i2, h2, fma(i3, h3, fma(-i0, h0, fma(-i1, h1, tz))));
    }
  } else {
    t = planar_inv_f64(r2, L2, L2x3);
    tz = t * dz;
  }
  const double w = pj.w * t;
  ax = fma(w, dx, ax);
  ay = fma(w, dy, ay);
  az = fma(pj.w, tz, az);
}

template <int MODE>
__device__ __forceinline__ void planar_tile_f64(const rd_d4* __restrict__ sj, int kmax, double x1,
                                                double y1, double z1, double qd1, int self_k,
                                                int nic, double d, int ic, double L2,
                                                double& ax, double& ay, double& az) {
  const float L2x3 = (float)(3.0 * L2);
  double tx = 0.0, ty = 0.0, tz = 0.0;
  for (int k = 0; k < kmax; ++k) {
    if (MODE == T_DIAG && k == self_k) continue;
    const bool upper = (MODE == T_UPPER) || (MODE == T_DIAG && k > self_k);
    planar_pair_f64(sj[k], x1, y1, z1, upper, nic, d, ic, L2, L2x3, tx, ty, tz);
  }
  ax = fma(qd1, tx, ax);
  ay = fma(qd1, ty, ay);
  az = fma(qd1, tz, az);
}

// ---- hyperboloid tip -------------------------------------------------------------
// Sphere image term (acc_tip_image_point.inc + acc_tip_ic_force.inc):
// a = lower-indexed particle, b = higher-indexed,
//   IC = K [ (a - b)/|b - a|^3 - c_a (im_a - b)/|b - im_a|^3 ],  c_a = R / dis_a,
// applied to the lower particle as is and to the higher one mirrored in x, y.
// With K = q0 / (4 pi eps0) ~ 1.4e-9 this part sits far below the FP32
// resolution of the direct sum, so the FP32 tiles keep it in separate sums
// that the caller scales by K in FP64.  For particle i against the j of one
// tile (d = x_i - x_j, e = image point - position):
//   D  = sum q d / |d|^3                          (all j; compensated d)
//   U  = sum_{j > i} q e_i / |e_i|^3,   e_i = im_i - x_j   (i in the a role)
//   W  = sum_{j < i} q c_j (ex, ey, -ez)_j / |e_j|^3,  e_j = im_j - x_i
//   Lz = sum_{j < i} q dz / |d|^3
// and the field is (1 + K) D + K (W - c_i U - 2 Lz z^).  U and W use the high
// words only: their relative error (~1e-5 for the nearest charges) is ~1e-14
// of the field once scaled by K.  MODE T_UPPER: every j in the a... b role of
// a point (fields), T_LOWER: every j lower, T_DIAG: by index against self_k.
struct TipSums {
  float dx, dy, dz, ux, uy, uz, wx, wy, wz, lz;
  __device__ void zero() { dx = dy = dz = ux = uy = uz = wx = wy = wz = lz = 0.f; }
};

// ELEC (off-diagonal tiles whose charges are all -1, the electrons' q/q0):
// the charge is a constant and its multiplies fold into the sums' signs.
template <int MODE, bool ELEC = false>
__device__ __forceinline__ void tip_tile_split_f32(const float4* __restrict__ sh, const float4* __restrict__ sl,
                                                   const float4* __restrict__ sih, int kmax, float4 ih,
                                                   float4 il, float4 iih, int self_k, int ic, TipSums& t) {
  for (int k = 0; k < kmax; ++k) {
    const float4 h = sh[k], l = sl[k];
    const float q = ELEC ? -1.f : ((MODE == T_DIAG && k == self_k) ? 0.f : h.w);
    const float dx = (ih.x - h.x) + (il.x - l.x);
    const float dy = (ih.y - h.y) + (il.y - l.y);
    const float dz = (ih.z - h.z) + (il.z - l.z);
    const float inv = rsqrtf(fmaf(dz, dz, fmaf(dx, dx, fmaf(dy, dy, 1e-20f))));
    const float s = q * ((inv * inv) * inv);
    t.dx = fmaf(s, dx, t.dx);
    t.dy = fmaf(s, dy, t.dy);
    t.dz = fmaf(s, dz, t.dz);
    if (ic) {
      const bool upper = (MODE == T_UPPER) || (MODE == T_DIAG && k > self_k);
      if (upper) {
        const float ex = iih.x - h.x, ey = iih.y - h.y, ez = iih.z - h.z;
        const float re = rsqrtf(fmaf(ez, ez, fmaf(ex, ex, fmaf(ey, ey, 1e-20f))));
        const float se = q * ((re * re) * re);
        t.ux = fmaf(se, ex, t.ux);
        t.uy = fmaf(se, ey, t.uy);
        t.uz = fmaf(se, ez, t.uz);
      } else {
        const float4 jh = sih[k];
        const float ex = jh.x - ih.x, ey = jh.y - ih.y, ez = jh.z - ih.z;
        const float re = rsqrtf(fmaf(ez, ez, fmaf(ex, ex, fmaf(ey, ey, 1e-20f))));
        const float se = (q * jh.w) * ((re * re) * re);
        t.wx = fmaf(se, ex, t.wx);
        t.wy = fmaf(se, ey, t.wy);
        t.wz = fmaf(-se, ez, t.wz);
        t.lz = fmaf(s, dz, t.lz);
      }
    }
  }
}

// The FP64 finish of the split sums: (1 + K) D + K (W - c_i U - 2 Lz z^), D
// given in FP64 (compensated across tiles), c_i = R / dis_i of the point.
__device__ __forceinline__ void tip_split_finish(double Dx, double Dy, double Dz, const TipSums& t, float ci,
                                                 int ic, double K, double* fx, double* fy, double* fz) {
  if (!ic) { *fx = Dx; *fy = Dy; *fz = Dz; return; }
  const double c = (double)ci;
  *fx = (1.0 + K) * Dx + K * ((double)t.wx - c * (double)t.ux);
  *fy = (1.0 + K) * Dy + K * ((double)t.wy - c * (double)t.uy);
  *fz = (1.0 + K) * Dz + K * (((double)t.wz - c * (double)t.uz) - 2.0 * (double)t.lz);
}

// FP64 tip gather: Calculate_Acceleration_Particles_ACC tip branch (:1344-1426),
// without the factor q_i k.  One pair (i, j); upper: i is the lower-indexed ("a")
// particle.  im: the image point of the "a" particle in the apex sphere and c = R /
// dis_a (tip_image_d4), the same for every pair a particle has that role in.  The
// image term's two distances to the power 3/2 are inverse cubes without the l^2, the
// first of them the Coulomb term's distance.  36 FP64 operations; with the image
// point formed per pair and pow(., 1.5) for the cubes a pair took several hundred.
__device__ __forceinline__ rd_d4 tip_image_d4(const DiodeParams& p, double xa, double ya, double za) {
  double xi, yi, zi;
  const double dis = tip_image_point(p, xa, ya, za, &xi, &yi, &zi);
  return make_d4(xi, yi, zi, p.r_tip / dis);
}
__device__ __forceinline__ void tip_pair_f64(const rd_d4& pj, const rd_d4& im, double x1, double y1, double z1,
                                             bool upper, int ic, double L2, float L2x3, double K, double& ax,
                                             double& ay, double& az) {
  const double dx = x1 - pj.x, dy = y1 - pj.y, dz = z1 - pj.z;
  const double r2 = fma(dz, dz, fma(dx, dx, dy * dy));
  double inv, ina;
  if (rd_cube_ok(r2)) {
    inv = rd_inv_cube<true>(r2, L2x3, &ina);
  } else {
    inv = rd_inv_cube_any(r2, L2);
    ina = rd_inv_cube_any(r2, 0.0);
  }
  if (!ic) {
    const double w = pj.w * inv;
    ax = fma(w, dx, ax); ay = fma(w, dy, ay); az = fma(w, dz, az);
    return;
  }
  // b: the particle that is not the "a" one.  x, y of the image term change sign for it.
  const double ex = im.x - (upper ? pj.x : x1), ey = im.y - (upper ? pj.y : y1), ez = im.z - (upper ? pj.z : z1);
  const double s2 = fma(ez, ez, fma(ex, ex, ey * ey));
  const double inb = rd_cube_ok(s2) ? rd_inv_cube0(s2) : rd_inv_cube_any(s2, 0.0);
  const double kb = K * (im.w * inb), ka = K * ina, kbs = upper ? kb : -kb;
  // upper: a - b = d; lower: a - b = -d, x and y mirrored
  const double wd = inv + ka, wz = upper ? wd : inv - ka;
  ax = fma(pj.w, fma(wd, dx, -(kbs * ex)), ax);
  ay = fma(pj.w, fma(wd, dy, -(kbs * ey)), ay);
  az = fma(pj.w, fma(wz, dz, -(kb * ez)), az);
}

// im1: the point's own image (it is the "a" particle of the pairs with j above);
// sim: the images of the tile's particles (not read in T_UPPER).
template <int MODE>
__device__ __forceinline__ void tip_tile_f64(const rd_d4* __restrict__ sj, const rd_d4* __restrict__ sim,
                                             const rd_d4& im1, int kmax, double x1, double y1, double z1, double qd1,
                                             int self_k, int ic, double L2, double K, double& ax, double& ay,
                                             double& az) {
  const float L2x3 = (float)(3.0 * L2);
  double tx = 0.0, ty = 0.0, tz = 0.0;
  for (int k = 0; k < kmax; ++k) {
    if (MODE == T_DIAG && k == self_k) continue;
    const bool upper = (MODE == T_UPPER) || (MODE == T_DIAG && k > self_k);
    tip_pair_f64(sj[k], upper ? im1 : sim[k], x1, y1, z1, upper, ic, L2, L2x3, K, tx, ty, tz);
  }
  ax = fma(qd1, tx, ax);
  ay = fma(qd1, ty, ay);
  az = fma(qd1, tz, az);
}
