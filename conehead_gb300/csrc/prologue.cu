// Fused beam prologue: voxel blocking -> radiological depth -> off-axis
// distance -> fluence -> softening/horn -> TERMA, one thread per voxel.
//
// Follows conehead/conehead.py:71-120 (cuda_hit_test), :209-254
// (cuda_d_eff with cuda_dda_3d :123-206), :286-314 (cuda_oad), :320-360
// (cuda_fluence), :641-655 (softening/horn, host numpy float32) and
// :364-377 (cuda_terma).  The reference runs these as six launches with a
// host round trip after each; here they are one pass over the grid that
// writes only TERMA (plus the intermediates when asked).
//
// Exactness: blocked, d_eff, oad, f_soften and f_horn reproduce the
// reference's rounding bit for bit (float32 with float64 where Numba
// promotes, no FMA contraction) where a call returns them; a dose-only call
// takes the off-axis distance from pairs of float32 (project_pairs) and adds a
// map's samples in pairs.  Blocking samples are classified with a float32
// projection first; a sample whose block cell is ambiguous within the voxel's
// error bound (lattice_centre; a fixed SAMPLE_DELTA on the general path) is
// recomputed with the exact float64 mirror, so GB300's low float64 rate is only
// paid at field edges.  Fluence and TERMA run in float32 (reference: float64
// fluence, float32 TERMA) and are compared with a tolerance.

#include <algorithm>
#include <cstdio>

#include "ch_internal.cuh"

namespace ch {

constexpr float SAMPLE_DELTA = 0.05f;   // cells (0.1 mm) of float32 slack of the general paths
// largest bound of a lattice sample's cell coordinates with which one neighbour
// per axis, on the sample's side of its cell, is all it may fall in (a bound
// below half a cell, less the roundings of the test)
constexpr float LATTICE_DELTA_MAX = 0.25f;

// partial sums 0, 1/27, 1/27+1/27, ... accumulated in float64 as the
// reference does for a block value of exactly 1.0 and 3x3x3 samples
__constant__ double c_unit_partial[28];
// for S = 1..16 sub-samples per axis: 1 / S^3, and the sum of S^3 such terms
__constant__ double c_inv_count[17];
__constant__ double c_unit_sum[17];

// --------------------------------------------------------- block lookup --
// cell index i = floor(100 x) (x in cm, beam coordinates); the reference
// reads block_values[i + 1999] after checking i + 2000 in [0, 3999]; index
// -1 wraps to the last row/column.
__device__ __forceinline__ float cell_value(const BeamDev& b, int fi, int fk) {
  const int c0 = fi + 2000, c1 = fk + 2000;
  if (c0 < 0 || c0 > 3999 || c1 < 0 || c1 > 3999) return 0.0f;
  int r = c0 - 1, c = c1 - 1;
  if (r < 0) r += b.full_rows;
  if (c < 0) c += b.full_cols;
  r -= b.br0;
  c -= b.bc0;
  if (r < 0 || r >= b.brows || c < 0 || c >= b.bcols) return 0.0f;
  if (b.uniform) return 1.0f;
  return __ldg(b.block + (size_t)r * b.bcols + c);
}

// floor of a float32 cell coordinate as the reference stores it; values far
// outside the map (and NaN) land outside [-2000, 1999], where every cell reads 0
__device__ __forceinline__ int floor_cell(float v) {
  if (!(v == v)) return 1 << 24;
  return (int)floorf(fminf(fmaxf(v, -1.0e7f), 1.0e7f));
}

// Exact projection, float64 source arrays (conehead.py:25-47 + :109-116).
__device__ __forceinline__ bool project_exact_mixed(const BeamDev& b, const float* rd, float& px,
                                                    float& pz) {
  const double ndotu =
      dadd(dadd(dmul(b.vy[0], (double)rd[0]), dmul(b.vy[1], (double)rd[1])), dmul(b.vy[2], (double)rd[2]));
  if (fabs(ndotu) < 1e-6) return false;
  const double si = ddiv(-b.vyw, ndotu);
  float pp[3];
#pragma unroll
  // (the reference adds the plane point 0 as well: it could only turn -0 into 0)
  for (int k = 0; k < 3; ++k) pp[k] = d2f(dadd(b.srcd[k], dmul(si, (double)rd[k])));
  px = d2f(dadd(dadd(dmul(b.m0[0], (double)pp[0]), dmul(b.m0[1], (double)pp[1])), dmul(b.m0[2], (double)pp[2])));
  pz = d2f(dadd(dadd(dmul(b.m2[0], (double)pp[0]), dmul(b.m2[1], (double)pp[1])), dmul(b.m2[2], (double)pp[2])));
  return true;
}

// Exact projection, float32 source arrays (all float32 arithmetic).
__device__ __forceinline__ bool project_exact_f32(const BeamDev& b, const float* rd, float& px,
                                                  float& pz) {
  const float ndotu = fadd(fadd(fmul(b.vyf[0], rd[0]), fmul(b.vyf[1], rd[1])), fmul(b.vyf[2], rd[2]));
  if (fabs((double)ndotu) < 1e-6) return false;
  const float si = fdiv(-b.vywf, ndotu);
  float pp[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) pp[k] = fadd(fadd(b.srcf[k], fmul(si, rd[k])), 0.0f);
  px = fadd(fadd(fmul(b.m0f[0], pp[0]), fmul(b.m0f[1], pp[1])), fmul(b.m0f[2], pp[2]));
  pz = fadd(fadd(fmul(b.m2f[0], pp[0]), fmul(b.m2f[1], pp[1])), fmul(b.m2f[2], pp[2]));
  return true;
}

// reference ray vector source - p, rounded to float32
__device__ __forceinline__ void ray_to_source(const BeamDev& b, const float* p, float* rd) {
  if (b.geom_f32) {
#pragma unroll
    for (int k = 0; k < 3; ++k) rd[k] = fsub(b.srcf[k], p[k]);
  } else {
#pragma unroll
    for (int k = 0; k < 3; ++k) rd[k] = d2f(dsub(b.src[k], (double)p[k]));
  }
}

// The float64 projection in pairs of float32 (48 bits): products with their
// exact residual, Knuth's two-sums, a quotient with one correction.  px and pz
// differ from project_exact_mixed's where that value lies within about 2^-46 of
// the terms of a float32 tie.  A float64 instruction holds the pipe of an SM quarter
// for 64 cycles, and the 33 of this projection were two thirds of what it did.
// Prologue, float64 / pairs: one beam at 64^3 29 / 24 us, 150 x 130 x 92 126 / 118, 32
// beams 5 x 5 cm at 128^3 441 / 423, 64 mixed beams 2686 / 2525, nine MLC beams 1048 /
// 988, seven at 192^3 (long walks) 457 / 459.  Intermediates keep the float64 bits.
struct Pair {
  float h, l;
};
__device__ __forceinline__ Pair two_sum(float a, float b) {
  const float s = fadd(a, b), bb = fsub(s, a);
  return {s, fadd(fsub(a, fsub(s, bb)), fsub(b, bb))};
}
__device__ __forceinline__ Pair pair_dot(const float* vh, const float* vl, const float* r) {
  Pair p[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    p[k].h = fmul(vh[k], r[k]);
    p[k].l = __fmaf_rn(vl[k], r[k], __fmaf_rn(vh[k], r[k], -p[k].h));
  }
  const Pair a = two_sum(p[0].h, p[1].h), t = two_sum(a.h, p[2].h);
  return {t.h, fadd(fadd(fadd(p[0].l, p[1].l), a.l), fadd(p[2].l, t.l))};
}
__device__ __forceinline__ bool project_pairs(const BeamDev& b, const float* rd, float& px, float& pz) {
  const Pair d = pair_dot(b.vyf, b.vyl, rd);
  const float h = fadd(d.h, d.l), l = fadd(fsub(d.h, h), d.l);
  if (!(fabsf(h) > 2e-6f)) return false;   // parallel, or nearly
  const float q1 = __fdividef(-b.vywh, h);
  const float q2 = __fdividef(fsub(__fmaf_rn(-q1, l, __fmaf_rn(-q1, h, -b.vywh)), b.vywl), h);
  float pp[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float m = fmul(q1, rd[k]), e = __fmaf_rn(q2, rd[k], __fmaf_rn(q1, rd[k], -m));
    const Pair s = two_sum(b.srcf[k], m);
    pp[k] = fadd(s.h, fadd(s.l, e));
  }
  const Pair x = pair_dot(b.m0f, b.m0l, pp), z = pair_dot(b.m2f, b.m2l, pp);
  px = fadd(x.h, x.l);
  pz = fadd(z.h, z.l);
  return true;
}

__device__ __forceinline__ bool project_exact(const BeamDev& b, const float* rd, float& px, float& pz) {
  return b.geom_f32 ? project_exact_f32(b, rd, px, pz) : project_exact_mixed(b, rd, px, pz);
}

// Exact transmission of one sub-sample (reference path end to end).  Kept
// out of line: it is rare, and inlining it at every sample site would bloat
// the kernel past the instruction cache.
// Block cell (floor(100 px), floor(100 pz)) of one sub-sample by the exact
// reference arithmetic; false (and bad = 1) for a ray parallel to the plane.
__device__ __forceinline__ bool sample_cell_exact(const BeamDev& b, const GridDev& g, const float* pos,
                                                  const float* off, int ix, int iy, int iz, int& bad, int& fi,
                                                  int& fk) {
  const int ii[3] = {ix, iy, iz};
  float ps[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    // ((pos - s/2) + off/2) + off*i, exact in float64 (a host check on the
    // grid's extent stands behind lat), one rounding
    const double v = b.lat ? __fma_rn((double)off[k], (double)((float)ii[k] + 0.5f),
                                      dsub((double)pos[k], (double)(g.spacing[k] * 0.5f)))
                           : dadd(dadd(dsub((double)pos[k], (double)g.spacing[k] * 0.5), (double)off[k] * 0.5),
                                  dmul((double)off[k], (double)ii[k]));
    ps[k] = d2f(v);
  }
  float rd[3];
  ray_to_source(b, ps, rd);
  float px, pz;
  if (!project_exact(b, rd, px, pz)) {
    bad = 1;
    return false;
  }
  fi = floor_cell(fmul(px, 100.0f));
  fk = floor_cell(fmul(pz, 100.0f));
  return true;
}

__device__ __noinline__ float sample_exact(const BeamDev& b, const GridDev& g, const float* pos, const float* off,
                              int ix, int iy, int iz, int& bad) {
  int fi, fk;
  if (!sample_cell_exact(b, g, pos, off, ix, iy, iz, bad, fi, fk)) return 0.0f;
  return cell_value(b, fi, fk);
}

// ------------------------------------------------------------ blocking --
// Transmission of sub-sample (ix, iy, iz) at pos + (rx, ry, rz) on the general
// path: float32 projection, exact float64 mirror only when the block cell is
// ambiguous within SAMPLE_DELTA.
__device__ __forceinline__ float sample_value(const BeamDev& b, const GridDev& g, const float* pos,
                                              const float* off, float rx, float ry, float rz, int ix, int iy,
                                              int iz, int& bad) {
  const float p0 = pos[0] + rx, p1 = pos[1] + ry, p2 = pos[2] + rz;
  const float np_ = b.vyf[0] * p0 + b.vyf[1] * p1 + b.vyf[2] * p2;
  const float m0p = b.m0f[0] * p0 + b.m0f[1] * p1 + b.m0f[2] * p2;
  const float m2p = b.m2f[0] * p0 + b.m2f[1] * p1 + b.m2f[2] * p2;
  const float ndr = b.a_nS - np_;
  // the float32 error bound assumes a magnification SAD/depth below 5; closer
  // to the source plane (or behind it) take the exact path, which also
  // reports rays parallel to the blocking plane as the reference does
  if (!(fabsf(ndr) > 0.2f * fabsf(b.a_K))) return sample_exact(b, g, pos, off, ix, iy, iz, bad);
  const float si = __fdividef(b.a_K, ndr);
  const float ux = (b.a_c0 + si * (b.a_m0S - m0p)) * 100.0f;
  const float uz = (b.a_c2 + si * (b.a_m2S - m2p)) * 100.0f;
  const int i0 = floor_cell(ux - SAMPLE_DELTA), i1 = floor_cell(ux + SAMPLE_DELTA);
  const int k0 = floor_cell(uz - SAMPLE_DELTA), k1 = floor_cell(uz + SAMPLE_DELTA);
  float v = cell_value(b, i0, k0);
  if (i0 != i1 || k0 != k1) {
    const float v1 = cell_value(b, i1, k0), v2 = cell_value(b, i0, k1), v3 = cell_value(b, i1, k1);
    if (v1 != v || v2 != v || v3 != v) v = sample_exact(b, g, pos, off, ix, iy, iz, bad);
  }
  return v;
}

// Whether the general paths must mirror every sample of a voxel: their fixed
// slack covers the float32 projection only where lattice_centre's bound, of the
// same terms in another order, is known and below half of it.
__device__ __noinline__ bool general_exact(const BeamDev& b, const float* pos);

// General blocked fraction, where the lattice below does not hold (float64,
// reference order acc = acc + v / S^3 over ix, iy, iz).
__device__ __noinline__ double blocked_general(const BeamDev& b, const GridDev& g, int S, const float* pos,
                                               int& bad) {
  float off[3];
  // f32(f64(s) / S) == fdiv(s, S): double rounding is innocuous for float32 operands
  for (int k = 0; k < 3; ++k) off[k] = fdiv(g.spacing[k], (float)S);
  const bool exact_all = general_exact(b, pos);
  double acc = 0.0;
  const double denom = (double)S * (double)S * (double)S;
  float last_v = -1.0f;
  double last_q = 0.0;
  for (int ix = 0; ix < S; ++ix)
    for (int iy = 0; iy < S; ++iy)
      for (int iz = 0; iz < S; ++iz) {
        float v;
        if (exact_all) {
          v = sample_exact(b, g, pos, off, ix, iy, iz, bad);
        } else {
          const float rx = off[0] * ((float)ix + 0.5f) - g.spacing[0] * 0.5f;
          const float ry = off[1] * ((float)iy + 0.5f) - g.spacing[1] * 0.5f;
          const float rz = off[2] * ((float)iz + 0.5f) - g.spacing[2] * 0.5f;
          v = sample_value(b, g, pos, off, rx, ry, rz, ix, iy, iz, bad);
        }
        if (v != last_v) {
          last_v = v;
          last_q = ddiv((double)v, denom);
        }
        acc = dadd(acc, last_q);
      }
  return acc;
}

// -------------------------------------------------- sub-sample lattice --
// The S^3 sub-samples are a lattice, so the three linear forms of the float32
// projection -- nd = n.(S - p), x0 = m0.(S - p), x2 = m2.(S - p) -- step by
// constants from sample to sample: a sample costs three FMAs, one fast
// reciprocal and two FMAs for its cell coordinates
//   u = 100 (c0 + K x0 / nd),   w = 100 (c2 + K x2 / nd),
// where the per-sample dot products cost about thirty instructions.
struct Centre {
  float nd, x0, x2;     // the linear forms at the voxel centre
  float u, w, mu, mw;   // its cell coordinates, and how far a sub-sample's may be from them
  float delta;          // bound of |float32 - reference| of a sample's cell coordinates
};

// Projects the voxel centre and bounds the sub-samples around it.  For an
// offset of the lattice's box, |d nd| <= A = lat_n, |d x0| <= B = lat_0, so
//   |d(K x0 / nd)| <= |K| (B + |x0 / nd| A) / (|nd| - A).
// False when a sub-sample may lie closer to the source plane than 0.2 |K| or
// may read the wrapped cell -2000 of a crop that holds the map's last row or
// column, or where delta is too large for a map's neighbour test: those voxels,
// and float32 source arrays, take blocked_general.
//
// delta bounds the difference between a float32 cell coordinate and the
// reference's, whose ray and plane point are float32 stores as well.  With
// P the largest |coordinate| of the grid, P1 the largest sum of three, D the
// largest distance to the source and m the magnification |K / nd|, in units of
// 2^-24 (a rounding of 1): the reference's sample point and ray are off by at
// most sqrt(3) P + D, which moves its plane point by m (1 + lat) times that;
// here x0 is off by 8 P1 + 5 |m0.S| (inputs, products, sums, lattice steps)
// and nd by 8 P1 + 5 |n.S|, which moves K x0 / nd by m and m lat times that.
// The plane point's own roundings, the quotient and the scaling by 100 stay
// below 0.002 cells within the map.  About 0.008 cells on a 40 cm grid: a
// seventh of the samples of a fixed 0.05 take the float64 mirror, which cost
// a map with graded cells (MLC leaf edges) two thirds of its TERMA launch.
__device__ __forceinline__ bool lattice_centre(const BeamDev& b, const float* pos, Centre& c) {
  if (!b.lat) return false;
  c.nd = b.a_nS - (b.vyf[0] * pos[0] + b.vyf[1] * pos[1] + b.vyf[2] * pos[2]);
  c.x0 = b.a_m0S - (b.m0f[0] * pos[0] + b.m0f[1] * pos[1] + b.m0f[2] * pos[2]);
  c.x2 = b.a_m2S - (b.m2f[0] * pos[0] + b.m2f[1] * pos[1] + b.m2f[2] * pos[2]);
  const float near = fabsf(c.nd) - b.lat_n;
  if (!(near > 0.2f * fabsf(b.a_K))) return false;
  const float K = 100.0f * b.a_K;
  const float inv = __fdividef(1.0f, c.nd), mag = __fdividef(fabsf(K), near);
  c.u = K * inv * c.x0 + 100.0f * b.a_c0;
  c.w = K * inv * c.x2 + 100.0f * b.a_c2;
  const float l0 = fabsf(c.x0 * inv), l2 = fabsf(c.x2 * inv);
  c.delta = mag * (b.err_x + (fmaxf(l0, l2) + 0.01f) * b.err_n) + 0.002f;
  c.mu = mag * (b.lat_0 + l0 * b.lat_n) + c.delta;
  c.mw = mag * (b.lat_2 + l2 * b.lat_n) + c.delta;
  if (!b.uniform && !(c.delta <= LATTICE_DELTA_MAX)) return false;
  return !b.wraps || (c.u - c.mu > -1999.0f && c.w - c.mw > -1999.0f);
}

// Takes its own look at the voxel: the general path is rare, and a bound handed
// to it cost 64 mixed beams 1% (registers of every voxel).
__device__ __noinline__ bool general_exact(const BeamDev& b, const float* pos) {
  Centre c;
  c.delta = 1.0e30f;
  lattice_centre(b, pos, c);       // leaves delta alone near the source plane and for float32 sources
  return !(c.delta <= 0.5f * SAMPLE_DELTA);
}

// Calls f(ix, iy, iz, u, w) for every sub-sample in the reference's order.  Rolled:
// three copies of a map lookup along z outgrew the instruction cache (nine MLC
// beams, prologue 1.23 -> 1.05 ms with five steps of the walk below instead of
// eight).
template <class F>
__device__ __forceinline__ void for_samples(const BeamDev& b, const float* off, int S, const Centre& c, F f) {
  const float K = 100.0f * b.a_K, c0 = 100.0f * b.a_c0, c2 = 100.0f * b.a_c2;
  const float mid = 0.5f * (float)(S - 1);
#pragma unroll 1
  for (int ix = 0; ix < S; ++ix) {
    const float rx = off[0] * ((float)ix - mid);
    const float nx = c.nd - b.vyf[0] * rx, x0x = c.x0 - b.m0f[0] * rx, x2x = c.x2 - b.m2f[0] * rx;
#pragma unroll 1
    for (int iy = 0; iy < S; ++iy) {
      const float ry = off[1] * ((float)iy - mid);
      const float ny = nx - b.vyf[1] * ry, x0y = x0x - b.m0f[1] * ry, x2y = x2x - b.m2f[1] * ry;
#pragma unroll 1
      for (int iz = 0; iz < S; ++iz) {
        const float rz = off[2] * ((float)iz - mid);
        const float si = __fdividef(K, ny - b.vyf[2] * rz);
        f(ix, iy, iz, si * (x0y - b.m0f[2] * rz) + c0, si * (x2y - b.m2f[2] * rz) + c2);
      }
    }
  }
}

// The 27 samples of a voxel (bit 26 - (9 ix + 3 iy + iz)) on one side of a line of
// the block map, u = edge or w = edge: sgn * (coordinate - edge) < 0.  The test
// K x0 / nd < h is a sign of K x0 - h nd, which is linear along the lattice: an
// add and a funnel shift per sample.  near gets the samples within the error
// bound of the line, which the caller decides exactly; the form's own rounding
// stays below 0.003 cells (six roundings of terms up to 2200 |nd|).
constexpr unsigned ALL_27 = 0x7ffffffu;
__device__ __forceinline__ unsigned below_edge(const BeamDev& b, const float* off, const Centre& c, bool along_u,
                                               float edge, float sgn, unsigned& near) {
  const float K = 100.0f * b.a_K;
  const float h = edge - 100.0f * (along_u ? b.a_c0 : b.a_c2);
  const float k = c.nd < 0.0f ? -sgn : sgn;
  const float kK = k * K, kh = k * h;
  float F = kK * (along_u ? c.x0 : c.x2) - kh * c.nd;
  const float* m = along_u ? b.m0f : b.m2f;
  const float fx = (kh * b.vyf[0] - kK * m[0]) * off[0], fy = (kh * b.vyf[1] - kK * m[1]) * off[1];
  const float fz = (kh * b.vyf[2] - kK * m[2]) * off[2];
  F -= fx + fy + fz;                                // sample (0, 0, 0)
  unsigned in = 0;
  float least = 3.0e38f;
#pragma unroll
  for (int ix = 0; ix < 3; ++ix)
#pragma unroll
    for (int iy = 0; iy < 3; ++iy) {
      const float f0 = F + ((float)ix * fx + (float)iy * fy);
#pragma unroll
      for (int iz = 0; iz < 3; ++iz) {
        const float f = f0 + (float)iz * fz;
        in = __funnelshift_l(__float_as_uint(f), in, 1);   // its sign bit into bit 0
        least = fminf(least, fabsf(f));
      }
    }
  const float tol = (c.delta + 0.003f) * (fabsf(c.nd) + b.lat_n);
  if (!(least > tol)) {
    unsigned n = 0;
#pragma unroll 1
    for (int ix = 0; ix < 3; ++ix)
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const float f = F + ((float)ix * fx + (float)(q / 3) * fy) + (float)(q % 3) * fz;
        n = (n << 1) | (fabsf(f) > tol ? 0u : 1u);
      }
    near |= n;
  }
  return in;
}

// Calls f(bit, ix, iy, iz) for every sample of a mask of below_edge's.
template <class F>
__device__ __forceinline__ void for_mask(unsigned mask, F f) {
  while (mask) {
    const int bit = __ffs(mask) - 1, i = 26 - bit;
    mask &= mask - 1;
    f(1u << bit, i / 9, (i / 3) % 3, i % 3);
  }
}

// Open samples (of 27) of a voxel that edges of a uniform crop cross (most
// voxels see one).
__device__ __forceinline__ int open_samples(const BeamDev& b, const GridDev& g, const float* pos, const float* off,
                                            const Centre& c, int& bad) {
  unsigned open = ALL_27, near = 0;
#pragma unroll 1
  for (int e = 0; e < 4; ++e) {
    const bool along_u = e < 2;
    const float sgn = (e & 1) ? -1.0f : 1.0f;
    const float edge = along_u ? b.uc + sgn * b.uh : b.wc + sgn * b.wh;
    if (fabsf((along_u ? c.u : c.w) - edge) <= (along_u ? c.mu : c.mw))
      open &= below_edge(b, off, c, along_u, edge, sgn, near);
  }
  for_mask(near, [&](unsigned bit, int ix, int iy, int iz) {
    open = sample_exact(b, g, pos, off, ix, iy, iz, bad) == 1.0f ? open | bit : open & ~bit;
  });
  return __popc(open);
}

// Adds every sub-sample's transmission by add(v): value(u, w, amb) gives it from
// the float32 coordinates or sets amb.  Ambiguous samples (up to 32 per voxel)
// are taken after the loop, one per lane and round, so that the exact path runs
// once or twice for a warp and not at every sample where one of its lanes needs
// it; add's order does not matter.
template <class V, class A>
__device__ __forceinline__ void add_samples(const BeamDev& b, const GridDev& g, const float* pos, const float* off,
                                            int S, const Centre& c, int& bad, V value, A add) {
  const bool defer = S <= 3;
  unsigned later = 0;
  for_samples(b, off, S, c, [&](int ix, int iy, int iz, float u, float w) {
    bool amb = false;
    float v = value(u, w, amb);
    if (amb) {
      if (defer) {
        later |= 1u << ((ix * S + iy) * S + iz);
        return;
      }
      v = sample_exact(b, g, pos, off, ix, iy, iz, bad);
    }
    add(v);
  });
  while (later) {
    const int i = __ffs(later) - 1;
    later &= later - 1;
    add(sample_exact(b, g, pos, off, i / (S * S), (i / S) % S, i % S, bad));
  }
}

// floor of a coordinate clamped to +-1e6, as an integer: adding 1.5 2^23
// rounding down leaves it in the low mantissa bits
__device__ __forceinline__ int floor_int(float v) {
  const float m = __fadd_rd(fminf(fmaxf(v, -1.0e6f), 1.0e6f), 12582912.0f);
  return __float_as_int(m) - 0x4b400000;
}

// transmission of cell (fi, fk); every cell here is past the wrapped one
__device__ __forceinline__ float map_value(const BeamDev& b, int fi, int fk) {
  const int r = fi + 1999 - b.br0, c = fk + 1999 - b.bc0;
  return ((unsigned)r < (unsigned)b.rlim && (unsigned)c < (unsigned)b.clim) ? __ldg(b.block + (size_t)r * b.bcols + c)
                                                                            : 0.0f;
}

// v / n correctly rounded for float32 v and n = S^3 <= 4096 without the
// division subroutine: product with the rounded reciprocal and one residual
// step (equal to the quotient for every float32 significand and S = 1..16,
// tests/test_lattice_cpu.py; infinities and NaN take the division)
__device__ __forceinline__ double div_count(float v, double n, double inv_n) {
  if (!(fabsf(v) <= 3.4028234e38f)) return ddiv((double)v, n);
  const double q = dmul((double)v, inv_n);
  return __fma_rn(__fma_rn(-n, q, (double)v), inv_n, q);
}

// Blocked fraction (float64, the reference's sum acc + v / S^3 over ix, iy,
// iz) of one voxel, every lane its own voxel.
//
// A uniform crop (jaws): a voxel whose samples all lie inside, or all outside,
// the open rectangle is decided by its centre and the lattice's bound; the
// others count their open samples by the signed distance to the rectangle
// (about 15 instructions a sample), and the sum of n ones and S^3 - n zeros
// is the n-th partial sum of 1 / S^3.  A map with other values looks every
// sample's cell up.  A sample within delta of a cell (or rectangle) edge that
// matters takes the exact float64 mirror.
//
// Both were bound by instruction issue: the field-edge voxels of a jaw field
// were classified one per warp round, 27 lanes each (a chunk of 32 edge voxels
// took 32 rounds), and a map's voxels went through those rounds and then again
// through a per-lane loop with a float64 division per change of value; then by
// float64 issue (sums, exact samples).  Prologues, start of that work / now:
// nine MLC beams on 140 x 101 x 112 8.59 / 0.87 ms, 64 mixed jaw beams 5.18 /
// 1.86 ms, 32 beams 5 x 5 cm on 128^3 0.88 / 0.31 ms (the walk, the projection and
// the cull have their share; this function alone, last step: 1.69 -> 1.22, 2.94 ->
// 2.69, 0.490 -> 0.446 ms).
//
// EXACT: the bits of the reference's float64 sum also for maps (where the
// blocked fraction itself is returned); otherwise their samples are added in
// 48 bits and divided once (5e-17 off on average, the float64 sum of quotients 1.4e-16).
// False where the general path must take the voxel.
template <bool EXACT>
__device__ __forceinline__ bool blocked_lattice(const BeamDev& b, const GridDev& g, int S, const float* pos, int& bad,
                                                double& blocked) {
  Centre c;
  if (!lattice_centre(b, pos, c)) return false;
  // signed distances (cells) of the centre outside the crop's open cells
  const float du = fabsf(c.u - b.uc) - b.uh, dw = fabsf(c.w - b.wc) - b.wh;
  blocked = 0.0;
  if (du > c.mu || dw > c.mw) return true;
  float off[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) off[k] = fdiv(g.spacing[k], (float)S);
  if (b.uniform) {
    if (du < -c.mu && dw < -c.mw) {
      blocked = c_unit_sum[S];
      return true;
    }
    if (S == 3) {
      blocked = c_unit_partial[open_samples(b, g, pos, off, c, bad)];
      return true;
    }
    int n = 0;
    add_samples(b, g, pos, off, S, c, bad,
                [&](float u, float w, bool& amb) {
                  const float d = fmaxf(fabsf(u - b.uc) - b.uh, fabsf(w - b.wc) - b.wh);
                  amb = fabsf(d) <= c.delta;
                  return d < 0.0f ? 1.0f : 0.0f;
                },
                [&](float v) { n += v == 1.0f ? 1 : 0; });
    const double q = c_inv_count[S];
    for (int i = 0; i < n; ++i) blocked = dadd(blocked, q);
    return true;
  }
  // Coordinates are within the crop and the bound around it: floor by the
  // magic addition needs no clamp.
  const float clear = 0.5f - c.delta;
  auto value = [&](float u, float w, bool& amb) {
    const float mu = __fadd_rd(u, 12582912.0f), mw = __fadd_rd(w, 12582912.0f);
    const int i = __float_as_int(mu) - 0x4b400000, k = __float_as_int(mw) - 0x4b400000;
    const float v = map_value(b, i, k);
    const float du = (u - (mu - 12582912.0f)) - 0.5f, dw = (w - (mw - 12582912.0f)) - 0.5f;
    if (fmaxf(fabsf(du), fabsf(dw)) >= clear) {
      const int i1 = fabsf(du) >= clear ? i + (du < 0.0f ? -1 : 1) : i;
      const int k1 = fabsf(dw) >= clear ? k + (dw < 0.0f ? -1 : 1) : k;
      const float v1 = map_value(b, i1, k), v2 = map_value(b, i, k1), v3 = map_value(b, i1, k1);
      amb = v1 != v || v2 != v || v3 != v;
    }
    return v;
  };
  const double count = (double)(S * S * S), inv = c_inv_count[S];
  if (EXACT) {
    // the reference's float64 sum, share by share (one value and its quotient kept)
    double acc = 0.0, q = 0.0;
    float last = 0.0f;
    for_samples(b, off, S, c, [&](int ix, int iy, int iz, float u, float w) {
      bool amb = false;
      float v = value(u, w, amb);
      if (amb) v = sample_exact(b, g, pos, off, ix, iy, iz, bad);
      if (v != last) {
        last = v;
        q = div_count(v, count, inv);
      }
      if (v != 0.0f) acc = dadd(acc, q);
    });
    blocked = acc;
    return true;
  }
  // ones are counted, other values summed in float32 pairs (48 bits, Knuth's
  // two-sum): float64 adds issue at two lanes per clock and SM
  int ones = 0;
  float hi = 0.0f, lo = 0.0f;
  add_samples(b, g, pos, off, S, c, bad, value, [&](float v) {
    ones += v == 1.0f ? 1 : 0;
    if (v != 0.0f && v != 1.0f) {
      const float t = fadd(hi, v), bb = fsub(t, hi);
      lo = fadd(lo, fadd(fsub(hi, fsub(t, bb)), fsub(v, bb)));
      hi = t;
    }
  });
  blocked = hi == 0.0f && lo == 0.0f && S == 3 ? c_unit_partial[ones]
                                               : ddiv(dadd(dadd((double)hi, (double)lo), (double)ones), count);
  // past float32's range (or an infinity or NaN in the map) the float64 sum decides
  return fabsf(hi) <= 3.4028234e38f;
}

// (one call site of the general path: a second one, for the sums past float32's
// range, cost nine MLC beams 0.4%)
template <bool EXACT>
__device__ __forceinline__ double blocked_fraction(const BeamDev& b, const GridDev& g, int S, const float* pos,
                                                   int& bad) {
  double blocked;
  return blocked_lattice<EXACT>(b, g, S, pos, bad, blocked) ? blocked : blocked_general(b, g, S, pos, bad);
}

// ------------------------------------------------------------------ DDA --
// radiological depth from voxel (x, y, z) toward the source (cuda_d_eff).
// The walk is generated UNROLL steps at a time so their density loads are
// in flight together; the float32 accumulation keeps the reference order.
// A step picks its axis with predicates, not branches: the lanes of a warp
// step along different axes, so three short branches cost every step all
// three paths (20 of 32 lanes active; TERMA of 32 beams at 128^3 638 -> 509 us,
// 547 -> 396 M warp instructions).  Also tried at 3 CTAs per SM: 4, 6 and 8
// steps with the next group's loads issued before this one's sums, 8 and 12 steps,
// and 64 registers (4 CTAs): all within 2%.
// The integer pipe, half as wide as the float32 one, then bound the issue (64%
// against 34% busy): steps left are counted in float32, their test and the
// smallest t are three-operand minima, the index advances by multiply-adds.
// Prologues: 32 beams at 128^3 334 -> 306 us, seven at 192^3 328 -> 295, 64 mixed
// 2055 -> 1862, nine MLC beams 904 -> 872, 150 x 130 x 92 108 -> 98.
constexpr int DDA_UNROLL = 5;

__device__ float radiological_depth(const float* __restrict__ rho, const GridDev& g, int x, int y, int z,
                                    const float* rd) {
  const float mag = __fsqrt_rn(fadd(fadd(fmul(rd[0], rd[0]), fmul(rd[1], rd[1])), fmul(rd[2], rd[2])));
  int s0, s1, s2;
  float t0, t1, t2, d0, d1, d2;
  dda_axis(fdiv(rd[0], mag), g.spacing[0], s0, t0, d0);
  dda_axis(fdiv(rd[1], mag), g.spacing[1], s1, t1, d1);
  dda_axis(fdiv(rd[2], mag), g.spacing[2], s2, t2, d2);
  const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
  // linear index of the density the reference reads at (x, y, z) and its
  // step along each grid axis (x and y swapped when swap_xy)
  // (volumes are limited to < 2^31 voxels by the host, so 32-bit indices)
  const int st0 = g.swap_xy ? n2 : n1 * n2;
  const int st1 = g.swap_xy ? n0 * n2 : n2;
  int idx = g.swap_xy ? (y * n0 + x) * n2 + z : (x * n1 + y) * n2 + z;
  const int dx = s0 * st0, dy = s1 * st1, dz = s2;
  // steps each axis may still take before the walk leaves the grid
  float left0 = (float)(s0 > 0 ? n0 - 1 - x : x), left1 = (float)(s1 > 0 ? n1 - 1 - y : y);
  float left2 = (float)(s2 > 0 ? n2 - 1 - z : z);
  auto inside = [&] { return fminf(fminf(left0, left1), left2) >= 0.0f; };
  int one = 1;
  asm volatile("" : "+r"(one));
  float deff = 0.0f, tprev = 0.0f;   // the first step adds rho * (t - 0), i.e. rho * t exactly
  // steps left are all >= 0 while the walk is inside the grid; an axis below 0
  // stays there.  A step past the exit reads no density and adds 0 * dt.
  // The axis with the smallest t steps, z before y before x where they tie.
  // one: 1 that the compiler does not know, so that the index sums are
  // multiply-adds (the float32 pipe) and not integer sums
  auto steps = [&](float (&r)[DDA_UNROLL], float (&tv)[DDA_UNROLL]) {
#pragma unroll
    for (int q = 0; q < DDA_UNROLL; ++q) {
      r[q] = inside() ? __ldg(rho + idx) : 0.0f;
      const float t = fminf(fminf(t0, t1), t2);
      tv[q] = t;
      asm("{\n .reg .pred p0, p1, p2;\n setp.le.f32 p2, %2, %7;\n setp.le.and.f32 p1|p0, %1, %7, !p2;\n"
          " @p0 add.rn.f32 %0, %0, %8;\n @p1 add.rn.f32 %1, %1, %9;\n @p2 add.rn.f32 %2, %2, %10;\n"
          " @p0 add.rn.f32 %3, %3, 0fBF800000;\n @p1 add.rn.f32 %4, %4, 0fBF800000;\n @p2 add.rn.f32 %5, %5, 0fBF800000;\n"
          " @p0 mad.lo.s32 %6, %14, %11, %6;\n @p1 mad.lo.s32 %6, %14, %12, %6;\n @p2 mad.lo.s32 %6, %14, %13, %6;\n}"
          : "+f"(t0), "+f"(t1), "+f"(t2), "+f"(left0), "+f"(left1), "+f"(left2), "+r"(idx)
          : "f"(t), "f"(d0), "f"(d1), "f"(d2), "r"(dx), "r"(dy), "r"(dz), "r"(one));
    }
  };
  auto add = [&](const float (&r)[DDA_UNROLL], const float (&tv)[DDA_UNROLL]) {
#pragma unroll
    for (int q = 0; q < DDA_UNROLL; ++q) {
      deff = fadd(deff, fmul(r[q], fsub(tv[q], tprev)));
      tprev = tv[q];
    }
  };
  while (inside()) {
    float r[DDA_UNROLL], tv[DDA_UNROLL];
    steps(r, tv);
    add(r, tv);
  }
  return deff;
}

// ------------------------------------------------------------ kernels --
// Whole-line rejection for the cull.  Along an (x, y) line the voxel centres
// lie on one segment.  While the depth stays positive, the projected
// coordinates xb(z), zb(z) and the lateral ratio are ratios of linear
// functions of z without a pole, hence monotone: their ranges over the line
// are spanned by the two end voxels, and 1/depth and the lateral ratio (and
// so the per-voxel margin) are bounded by their largest end values.  Depth
// is linear, so its minimum is at an end too.  True only when no voxel of
// the line can pass the per-voxel test below; 0.01 cm on top of the margin
// covers the float32 rounding of both tests (about 1e-5 cm here).
__device__ __forceinline__ bool line_outside(const GridDev& g, const BeamDev& b, float px, float py) {
  // every lane of the warp tests the same line: even lanes project its first
  // voxel, odd lanes its last, and one shuffle step combines the two
  const unsigned full = 0xffffffffu;
  const int e = threadIdx.x & 1;
  const float kk = fabsf(b.a_K);
  const float pz = voxel_centre(g.origin[2], g.spacing[2], e ? g.n[2] - 1 : 0);
  const float np_ = b.vyf[0] * px + b.vyf[1] * py + b.vyf[2] * pz;
  const float m0p = b.m0f[0] * px + b.m0f[1] * py + b.m0f[2] * pz;
  const float m2p = b.m2f[0] * px + b.m2f[1] * py + b.m2f[2] * pz;
  const float depth = np_ - b.a_nS;
  const bool ok = depth > 0.2f * kk;
  // near or behind the source plane at either end: test per voxel
  if (!(ok && __shfl_xor_sync(full, (int)ok, 1))) return false;
  const float inv = 1.0f / depth;
  const float si = -b.a_K * inv;
  const float xb = b.a_c0 + si * (b.a_m0S - m0p);
  const float zb = b.a_c2 + si * (b.a_m2S - m2p);
  const float lat = fmaxf(fabsf(b.a_m0S - m0p), fabsf(b.a_m2S - m2p)) * inv;
  const float xb2 = __shfl_xor_sync(full, xb, 1), zb2 = __shfl_xor_sync(full, zb, 1);
  const float inv_max = fmaxf(inv, __shfl_xor_sync(full, inv, 1));
  const float lat_max = fmaxf(lat, __shfl_xor_sync(full, lat, 1));
  const float xlo = fminf(xb, xb2), xhi = fmaxf(xb, xb2), zlo = fminf(zb, zb2), zhi = fmaxf(zb, zb2);
  const float M = b.cull_margin_k * kk * inv_max * (1.0f + lat_max) + 0.02f;
  return xhi < b.cx_lo - M || xlo > b.cx_hi + M || zhi < b.cz_lo - M || zlo > b.cz_hi + M;
}

// Whether the beam may reach the voxel centred at pos: its projection against
// the opening widened by the sub-samples' margin.
__device__ __forceinline__ bool cull_candidate(const BeamDev& b, const float* pos) {
  if (!b.cull_enable) return true;
  const float np_ = b.vyf[0] * pos[0] + b.vyf[1] * pos[1] + b.vyf[2] * pos[2];
  const float m0p = b.m0f[0] * pos[0] + b.m0f[1] * pos[1] + b.m0f[2] * pos[2];
  const float m2p = b.m2f[0] * pos[0] + b.m2f[1] * pos[1] + b.m2f[2] * pos[2];
  const float depth = np_ - b.a_nS;   // -n . (S - p)
  if (!(depth > 0.2f * fabsf(b.a_K))) return true;
  // one fast reciprocal: its ~2 ulp error is far inside the 0.01 cm
  // margin, so the candidate set stays a superset of the beam
  const float inv_depth = __fdividef(1.0f, depth);
  const float si = -b.a_K * inv_depth;
  const float xb = b.a_c0 + si * (b.a_m0S - m0p);
  const float zb = b.a_c2 + si * (b.a_m2S - m2p);
  const float lat = fmaxf(fabsf(b.a_m0S - m0p), fabsf(b.a_m2S - m2p)) * inv_depth;
  const float margin = b.cull_margin_k * fabsf(b.a_K) * inv_depth * (1.0f + lat) + 0.01f;
  return !(xb < b.cx_lo - margin || xb > b.cx_hi + margin || zb < b.cz_lo - margin || zb > b.cz_hi + margin);
}

// Pass 1, every voxel: zero TERMA and keep the voxels the beam may reach
// (all voxels when intermediates are requested) on a compact list, so the
// blocking/depth/TERMA pass runs on full warps.
// One warp per (x, y) line of the grid, lanes along z: the index arithmetic
// runs once per line and the zeroing of TERMA is coalesced.
__device__ __forceinline__ void cull_line(const GridDev& g, const BeamDev& b, float* __restrict__ T,
                                          const Inter& inter, int all_voxels, int* __restrict__ list_count,
                                          int* __restrict__ list_v, int line) {
  // volumes hold fewer than 2^31 voxels (checked on the host)
  if (line >= g.n[0] * g.n[1]) return;   // whole warp
  const int lane = threadIdx.x & 31;
  const int x = line / g.n[1], y = line - x * g.n[1];
  const float px = voxel_centre(g.origin[0], g.spacing[0], x);
  const float py = voxel_centre(g.origin[1], g.spacing[1], y);
  float* Tl = T + ((size_t)x * g.n[1] + y) * g.zp;
  // a line the beam cannot reach lists nothing (intermediates of every voxel
  // are written by the per-voxel loop, so it runs whenever they are asked)
  const bool no_inter = !inter.blocked && !inter.d_eff && !inter.oad && !inter.fluence && !inter.f_soften &&
                        !inter.f_horn && !inter.terma;
  if (b.cull_enable && !all_voxels && no_inter && line_outside(g, b, px, py)) {
    for (int z = lane; z < g.n[2]; z += 32) Tl[z] = 0.0f;
    return;
  }
  for (int z0 = 0; z0 < g.n[2]; z0 += 32) {
    const int z = z0 + lane;
    const bool live = z < g.n[2];
    const int v = line * g.n[2] + z;
    bool keep = false;
    if (live) {
      float pos[3];
      pos[0] = px;
      pos[1] = py;
      pos[2] = voxel_centre(g.origin[2], g.spacing[2], z);
      const bool candidate = cull_candidate(b, pos);
      keep = candidate || all_voxels;
      Tl[z] = 0.0f;
      if (!keep) {
        if (inter.blocked) inter.blocked[v] = 0.0;
        if (inter.d_eff) inter.d_eff[v] = 0.0f;
        if (inter.oad) inter.oad[v] = 0.0f;
        if (inter.fluence) inter.fluence[v] = 0.0f;
        if (inter.f_soften) inter.f_soften[v] = 1.0f;
        if (inter.f_horn) inter.f_horn[v] = 1.0f;
        if (inter.terma) inter.terma[v] = 0.0f;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    if (m) {
      int base = 0;
      if (lane == 0) base = atomicAdd(list_count, __popc(m));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (keep) list_v[base + __popc(m & ((1u << lane) - 1u))] = v;
    }
  }
}

__global__ void __launch_bounds__(256) cull_kernel(GridDev g, BeamDev b, float* __restrict__ T, Inter inter,
                                                   int all_voxels, int* __restrict__ list_count,
                                                   int* __restrict__ list_v) {
  cull_line(g, b, T, inter, all_voxels, list_count, list_v, (blockIdx.x * blockDim.x + threadIdx.x) >> 5);
}

// this CTA's beam record (blockIdx.y) copied into shared memory
__device__ __forceinline__ void load_record(const PrologueBeam* __restrict__ recs, PrologueBeam& R) {
  static_assert(sizeof(PrologueBeam) % 4 == 0 && sizeof(PrologueBeam) <= 4 * 1024, "record copy");
  const int* src = reinterpret_cast<const int*>(recs + blockIdx.y);
  int* dst = reinterpret_cast<int*>(&R);
  for (int i = threadIdx.x; i < (int)(sizeof(PrologueBeam) / 4); i += blockDim.x) dst[i] = __ldg(src + i);
  __syncthreads();
}

// Voxels [x, y) of a line that the beam may reach: line_outside's argument,
// solved for z.  With depth, x0 and x2 linear along the line, "xb >= cx_lo - M"
// times depth, M the line's largest margin, is linear too: its end values say
// whether it holds everywhere, nowhere or up to a crossing.  A line that comes
// near the source plane is kept whole.  A NaN restricts nothing.
__device__ __forceinline__ int2 line_span(const GridDev& g, const BeamDev& b, float px, float py) {
  const int nz = g.n[2];
  if (!b.cull_enable) return make_int2(0, nz);
  const float kk = fabsf(b.a_K);
  const float n_xy = b.vyf[0] * px + b.vyf[1] * py, x0_xy = b.a_m0S - (b.m0f[0] * px + b.m0f[1] * py);
  const float x2_xy = b.a_m2S - (b.m2f[0] * px + b.m2f[1] * py);
  float depth[2], x0[2], x2[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float pz = voxel_centre(g.origin[2], g.spacing[2], e ? nz - 1 : 0);
    depth[e] = (n_xy + b.vyf[2] * pz) - b.a_nS;
    x0[e] = x0_xy - b.m0f[2] * pz;
    x2[e] = x2_xy - b.m2f[2] * pz;
  }
  if (!(depth[0] > 0.2f * kk && depth[1] > 0.2f * kk)) return make_int2(0, nz);
  const float i0 = 1.0f / depth[0], i1 = 1.0f / depth[1];
  const float lat = fmaxf(fmaxf(fabsf(x0[0]), fabsf(x2[0])) * i0, fmaxf(fabsf(x0[1]), fabsf(x2[1])) * i1);
  const float M = b.cull_margin_k * kk * fmaxf(i0, i1) * (1.0f + lat) + 0.02f;
  float lo = 0.0f, hi = (float)(nz - 1);
  bool none = false;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float* v = k < 2 ? x0 : x2;
    const float c = k < 2 ? b.a_c0 : b.a_c2;
    const float edge = k == 0 ? b.cx_lo : k == 1 ? b.cx_hi : k == 2 ? b.cz_lo : b.cz_hi;
    const float w = (k & 1) ? (edge - c) + M : (c - edge) + M, K = (k & 1) ? b.a_K : -b.a_K;
    const float g0 = w * depth[0] + K * v[0], g1 = w * depth[1] + K * v[1];
    none = none || (g0 < 0.0f && g1 < 0.0f);
    const float t = g0 / (g0 - g1) * (float)(nz - 1);
    if (g0 < 0.0f && g1 >= 0.0f) lo = fmaxf(lo, t - 0.01f);
    if (g1 < 0.0f && g0 >= 0.0f) hi = fminf(hi, t + 0.01f);
  }
  const int z0 = max((int)ceilf(lo), 0), z1 = min((int)floorf(hi), nz - 1) + 1;
  return none || z1 <= z0 ? make_int2(0, 0) : make_int2(z0, z1);
}

// Every beam of a batch in one launch (blockIdx.y = beam), lpw lines per warp (at
// most 32), one per lane: its span of voxels, one add to the beam's list count
// for the whole warp, then line by line the list entries and, where only these
// lines are read, TERMA's zeros in 16-byte stores.
//
// Issue bound at first: a warp per line, a projection per voxel and an add, whose
// result it waited for, per 32 voxels / lane pairs testing lines and the
// projections on those that passed (230 instructions per 32 voxels, 83% issue
// active) / this, which writes 8 bytes per listed voxel: 32 beams at 128^3 157 / 75 /
// 30 us, seven at 192^3 130 / 100 / 19, 64 mixed beams 671 / 305 / 63.  The TERMA launch
// gained too, its chunks running along lines in order (64 mixed beams 2.22 -> 1.98
// ms).  Prologues, last step: 424 -> 332 us, 457 -> 328, 2523 -> 2050.
__global__ void __launch_bounds__(256) cull_batch_kernel(const PrologueBeam* __restrict__ recs, int lpw) {
  __shared__ PrologueBeam R;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  after_trigger();
  after_wait();
  {
    const PrologueBeam& G = recs[blockIdx.y];
    if ((int)(blockIdx.x * (blockDim.x >> 5)) * lpw >= G.g.n[0] * G.g.n[1]) return;   // whole CTA
  }
  load_record(recs, R);
  const GridDev& g = R.g;
  const int n1 = g.n[1], nz = g.n[2], lines = g.n[0] * n1, quads = g.zp >> 2;
  const int line0 = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * lpw;
  const int mine = min(lpw, lines - line0);    // this warp's lines
  if (mine <= 0) return;                       // whole warp
  const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  int2 span = make_int2(0, 0);
  if (lane < mine) {
    const int line = line0 + lane, x = line / n1, y = line - x * n1;
    span = line_span(g, R.b, voxel_centre(g.origin[0], g.spacing[0], x), voxel_centre(g.origin[1], g.spacing[1], y));
    R.line_any[line] = span.y > span.x ? 1 : 0;
  }
  if (R.zero_all) {                            // the gather reads TERMA anywhere
    float4* T4 = reinterpret_cast<float4*>(R.T + (size_t)line0 * g.zp);
    for (int e = lane; e < mine * quads; e += 32) T4[e] = zero;
  }
  const int count = span.y - span.x;
  int incl = count;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += up;
  }
  const int total = __shfl_sync(full, incl, 31);
  if (total == 0) return;
  int base = 0;
  if (lane == 0) base = atomicAdd(R.aabb + 6, total);
  base = __shfl_sync(full, base, 0) + incl - count;
  for (unsigned m = __ballot_sync(full, count > 0); m; m &= m - 1) {
    const int l = __ffs(m) - 1, line = line0 + l;
    const int n = __shfl_sync(full, count, l), v = line * nz + __shfl_sync(full, span.x, l);
    int* dst = R.list_v + __shfl_sync(full, base, l);
    for (int i = lane; i < n; i += 32) dst[i] = v + i;
    if (!R.zero_all) {
      float4* T4 = reinterpret_cast<float4*>(R.T + (size_t)line * g.zp);
      for (int e = lane; e < quads; e += 32) T4[e] = zero;
    }
  }
}

// TERMA of voxel (x, y, z) centred at pos, v its index: blocked fraction, then
// (where the beam is not fully blocked, or for every voxel when intermediates
// are requested) radiological depth, oad, fluence, softening/horn and TERMA.
// False when the voxel is blocked and nothing is written (Tv = 0).
template <bool EXACT>
__device__ __forceinline__ bool terma_voxel(const float* __restrict__ rho, const GridDev& g, const BeamDev& b,
                                            const SettingsDev& s, const Inter& inter, int all_voxels, int x, int y,
                                            int z, int v, const float* pos, int& bad, float& Tv) {
  Tv = 0.0f;
  const double blocked = blocked_fraction<EXACT>(b, g, s.samples, pos, bad);
  if (inter.blocked) inter.blocked[v] = blocked;
  if (blocked == 0.0 && !all_voxels) {
    if (inter.terma) inter.terma[v] = 0.0f;
    return false;
  }
  float rd[3];
  ray_to_source(b, pos, rd);
  // ---- radiological depth (float32, exact mirror)
  const float deff = radiological_depth(rho, g, x, y, z, rd);
  // ---- off-axis distance (exact mirror)
  float px = 0.0f, pz = 0.0f;
  if (EXACT || !b.pairs || !project_pairs(b, rd, px, pz))
    if (!project_exact(b, rd, px, pz)) bad = 1;
  const float oad = __fsqrt_rn(fadd(fmul(px, px), fmul(pz, pz)));
  // ---- fluence (float32 evaluation of the reference's float64 formula)
  const float mag = __fsqrt_rn(fadd(fadd(fmul(rd[0], rd[0]), fmul(rd[1], rd[1])), fmul(rd[2], rd[2])));
  const float sad = (float)b.sad;
  const float ratio = sad / mag;
  const float fpoint = s.sPri * (ratio * ratio);
  const float r_ann = oad * s.zAnn / sad;
  float fann = 0.0f;
  if (r_ann >= s.rInner && r_ann <= s.rOuter) {
    const float a = sad - s.zAnn, c = mag - s.zAnn;
    fann = s.sAnn * (a * a) / (c * c);
  }
  const float oadc = oad < 2.0f ? 2.0f : oad;
  const float r_exp = oadc * s.zExp / sad;
  const float ae = sad - s.zExp, ce = mag - s.zExp;
  const float fexp = s.sExp / r_exp * expf(-s.kExp * r_exp) * (ae * ae) / (ce * ce);
  // a product with the sum of S^3 equal shares (1 within a few 2^-53) rounds
  // to the float32 factor itself
  const bool open = blocked == c_unit_sum[s.samples];
  float fluence = fpoint + fann + fexp;
  if (!open) fluence = (float)((double)fluence * blocked);
  // ---- softening and horn (reference host numpy, float32)
  float fs = 1.0f;
  if (oad < s.softLimit) fs = fdiv(1.0f, fsub(1.0f, fmul(s.softRatio, oad)));
  const float fh = fadd(1.0f, fmul(oad, s.hornRatio));
  // ---- TERMA (float32, reference order)
  float terma = 0.0f;
  for (int i = 0; i < s.n_energy; ++i) {
    const float ex = expf(fmul(fmul(-s.mu[i], fs), deff));
    terma = fadd(terma, fmul(fmul(fmul(fmul(fmul(s.w[i], fluence), ex), s.E[i]), s.mu[i]), fh));
  }
  Tv = open ? terma : d2f(dmul((double)terma, blocked));
  if (inter.d_eff) inter.d_eff[v] = deff;
  if (inter.oad) inter.oad[v] = oad;
  if (inter.fluence) inter.fluence[v] = fluence;
  if (inter.f_soften) inter.f_soften[v] = fs;
  if (inter.f_horn) inter.f_horn[v] = fh;
  if (inter.terma) inter.terma[v] = Tv;
  return true;
}

// Pass 2, listed voxels (EXACT: all voxels in order where there is no list):
// TERMA and its support box for the cone stage.
// Entry e of a beam's list of count voxels; every lane of the warp calls it
// (the box reduction is warp-wide).
template <bool EXACT>
__device__ __forceinline__ void terma_entry(const float* __restrict__ rho, const GridDev& g, const BeamDev& b,
                                            const SettingsDev& s, float* __restrict__ T, const Inter& inter,
                                            int all_voxels, int count, unsigned e, const int* __restrict__ list_v,
                                            int* __restrict__ aabb, int* __restrict__ flags) {
  {
    const bool live = e < (unsigned)count;
    int x = 0, y = 0, z = 0, bad = 0;
    float Tv = 0.0f;
    if (live) {
      const int v = EXACT && !list_v ? (int)e : list_v[e];
      z = v % g.n[2];
      const int r = v / g.n[2];
      y = r % g.n[1];
      x = r / g.n[1];
      const float pos[3] = {voxel_centre(g.origin[0], g.spacing[0], x), voxel_centre(g.origin[1], g.spacing[1], y),
                            voxel_centre(g.origin[2], g.spacing[2], z)};
      if (terma_voxel<EXACT>(rho, g, b, s, inter, all_voxels, x, y, z, v, pos, bad, Tv))
        T[((size_t)x * g.n[1] + y) * g.zp + z] = Tv;
    }
    // ---- support box of T != 0 (the reference skips T == 0 sources), for the
    // gather's tap ranges.  Its six words share one L2 sector, and every chunk
    // of a beam in flight updated them: those adds took a sixth of the launch
    // (64 mixed beams, TERMA 3.20 -> 2.69 ms without them; with the walk, the
    // blocking and the spectrum left out they were three quarters of it).  The
    // spectral method needs no box, and a chunk inside the box so far adds
    // nothing.
    if (aabb) {
      const bool nz_ = live && Tv != 0.0f;
      if (__any_sync(0xffffffffu, nz_)) {
        const int lo0 = __reduce_min_sync(0xffffffffu, nz_ ? x : INT_MAX);
        const int hi0 = __reduce_max_sync(0xffffffffu, nz_ ? x : INT_MIN);
        const int lo1 = __reduce_min_sync(0xffffffffu, nz_ ? y : INT_MAX);
        const int hi1 = __reduce_max_sync(0xffffffffu, nz_ ? y : INT_MIN);
        const int lo2 = __reduce_min_sync(0xffffffffu, nz_ ? z : INT_MAX);
        const int hi2 = __reduce_max_sync(0xffffffffu, nz_ ? z : INT_MIN);
        if ((threadIdx.x & 31) == 0) {
          if (lo0 < __ldcg(aabb + 0)) atomicMin(aabb + 0, lo0);
          if (hi0 > __ldcg(aabb + 1)) atomicMax(aabb + 1, hi0);
          if (lo1 < __ldcg(aabb + 2)) atomicMin(aabb + 2, lo1);
          if (hi1 > __ldcg(aabb + 3)) atomicMax(aabb + 3, hi1);
          if (lo2 < __ldcg(aabb + 4)) atomicMin(aabb + 4, lo2);
          if (hi2 > __ldcg(aabb + 5)) atomicMax(aabb + 5, hi2);
        }
      }
    }
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flags, FLAG_PARALLEL_RAY);
  }
}

// The listed voxels of one beam, taken by n_ctas CTAs (this one is cta) in
// rounds of n_ctas * blockDim.x.
__device__ __forceinline__ void terma_body(const float* __restrict__ rho, const GridDev& g, const BeamDev& b,
                                           const SettingsDev& s, float* __restrict__ T, const Inter& inter,
                                           int all_voxels, const int* __restrict__ list_count,
                                           const int* __restrict__ list_v, int* __restrict__ aabb,
                                           int* __restrict__ flags, int cta, int n_ctas) {
  const int count = list_v ? *list_count : g.n[0] * g.n[1] * g.n[2];
  const unsigned stride = blockDim.x * n_ctas, rounds = ((unsigned)count + stride - 1) / stride;
  for (unsigned it = 0; it < rounds; ++it)
    terma_entry<true>(rho, g, b, s, T, inter, all_voxels, count, (it * n_ctas + cta) * blockDim.x + threadIdx.x,
                list_v, aabb, flags);
}

__global__ void __launch_bounds__(256) terma_kernel(const float* __restrict__ rho, GridDev g, BeamDev b,
                                                    SettingsDev s, float* __restrict__ T, Inter inter,
                                                    int all_voxels, const int* __restrict__ list_count,
                                                    const int* __restrict__ list_v, int* __restrict__ aabb,
                                                    int* __restrict__ flags) {
  terma_body(rho, g, b, s, T, inter, all_voxels, list_count, list_v, aabb, flags, blockIdx.x, gridDim.x);
}

// Every beam's listed voxels in one launch, in chunks of 32 (one per lane)
// that warps claim from one counter: claim c is chunk c - base of the beam
// whose chunks cover c, where base counts the chunks of the beams before it
// (entries 32 (c - base) .. 32 (c - base) + 31 of its list).  A warp that finishes
// early takes the next chunk of any beam, so the SMs end together however
// unequal the beams' lists and ray lengths are (a static share per CTA left
// the SMs idle for a sixth of the launch).  Each warp keeps the record of
// its current beam in its own shared slot and copies the next one when the
// claimed chunk moves on to another beam; the claims of one warp increase,
// so the beam search walks forward only.
constexpr int TERMA_WARPS = 8;   // 256 threads

__global__ void __launch_bounds__(256, 3) terma_batch_kernel(const PrologueBeam* __restrict__ recs, int n_beams,
                                                          int* __restrict__ flags, int* __restrict__ work) {
  __shared__ PrologueBeam Rw[TERMA_WARPS];
  static_assert(sizeof(PrologueBeam) % 4 == 0, "record copy");
  const int lane = threadIdx.x & 31;
  PrologueBeam& R = Rw[threadIdx.x >> 5];
  int cur = -1, beam = 0, base = 0, count = 0;
  after_trigger();
  after_wait();
  for (;;) {
    int c = 0;
    if (lane == 0) c = atomicAdd(work, 1);
    c = __shfl_sync(0xffffffffu, c, 0);
    // chunks of beam b: ceil(list count / 32); the counts were written by the cull launch
    while (beam < n_beams) {
      count = recs[beam].aabb[6];
      const int chunks = list_chunks(count);
      if (c < base + chunks) break;
      base += chunks;
      ++beam;
    }
    if (beam >= n_beams) break;   // whole warp
    if (beam != cur) {
      __syncwarp();
      const int* src = reinterpret_cast<const int*>(recs + beam);
      int* dst = reinterpret_cast<int*>(&R);
      for (int i = lane; i < (int)(sizeof(PrologueBeam) / 4); i += 32) dst[i] = __ldg(src + i);
      __syncwarp();
      cur = beam;
    }
    terma_entry<false>(R.rho, R.g, R.b, R.s, R.T, Inter{}, 0, count, ((c - base) << 5) + lane, R.list_v,
                R.box ? R.aabb : nullptr, flags);
  }
}

// Cull and TERMA of a few small beams in one launch, a warp per (x, y) line:
// the span of its candidate voxels, then TERMA of the span 32 voxels at a time and zeros beside it (on lines without candidates nothing:
// line_any says so).  No list, no counters to reset, and the records come as a
// kernel parameter: where the beams' voxels do not fill the SMs for long, the
// time is that of launches and of one chunk's latency, and this needs one
// launch and no copy instead of three and one.  flag_word gets the call's
// epoch where a ray is parallel to the blocking plane.
__global__ void __launch_bounds__(256, 3) prologue_fused_kernel(const __grid_constant__ FusedRecords A, int* flag_word,
                                                                int epoch) {
  const PrologueBeam& R = A.r[blockIdx.y];
  const GridDev& g = R.g;
  const BeamDev& b = R.b;
  const int line = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  after_trigger();
  after_wait();
  if (line >= g.n[0] * g.n[1]) return;   // whole warp
  const int x = line / g.n[1], y = line - x * g.n[1], nz = g.n[2];
  float pos[3] = {voxel_centre(g.origin[0], g.spacing[0], x), voxel_centre(g.origin[1], g.spacing[1], y), 0.0f};
  const int2 span = line_span(g, b, pos[0], pos[1]);
  const int lo = span.x, hi = span.y - 1;
  if (lane == 0) R.line_any[line] = hi >= lo;
  if (hi < lo) return;
  float* const T = R.T + (size_t)line * g.zp;
  for (int z = lane; z < lo; z += 32) T[z] = 0.0f;
  int bad = 0;
  for (int z = lo + lane; z - lane <= hi; z += 32) {
    float Tv = 0.0f;
    pos[2] = voxel_centre(g.origin[2], g.spacing[2], z);
    if (z <= hi) terma_voxel<false>(R.rho, g, b, R.s, Inter{}, 0, x, y, z, 0, pos, bad, Tv);
    if (z < nz) T[z] = Tv;
    __syncwarp();
  }
  const int end = lo + (hi - lo) / 32 * 32 + 32;
  for (int z = end + lane; z < nz; z += 32) T[z] = 0.0f;
  if (__any_sync(0xffffffffu, bad) && lane == 0) *flag_word = epoch;
}

void launch_prologue_fused(const FusedRecords& recs, int n_beams, long long max_lines, int* flag_word, int epoch,
                           cudaStream_t st) {
  launch_after(true, prologue_fused_kernel, dim3((unsigned)((max_lines + 7) / 8), n_beams), 256, 0, st, recs, flag_word, epoch);
}

// ----------------------------------------------------- beamlet adjoint --
// Beamlet holding block cell (fi, fk) under the lookup rule of cell_value
// (cell + 1999, index -1 wrapping to the last row/column), or -1.
__device__ __forceinline__ int beamlet_of(const BeamDev& b, const BeamletDev& bl, int fi, int fk) {
  const int c0 = fi + 2000, c1 = fk + 2000;
  if (c0 < 0 || c0 > 3999 || c1 < 0 || c1 > 3999) return -1;
  int r = c0 - 1, c = c1 - 1;
  if (r < 0) r += b.full_rows;
  if (c < 0) c += b.full_cols;
  r -= bl.r0;
  c -= bl.c0;
  if (r < 0 || c < 0 || r >= bl.rows * bl.cell_rows || c >= bl.cols * bl.cell_cols) return -1;
  return (r / bl.cell_rows) * bl.cols + c / bl.cell_cols;
}

// Beamlet of sub-sample (ix, iy, iz): the float32 projection decides when
// every cell within SAMPLE_DELTA of it lies in one beamlet, otherwise (or
// where exact says that the bound may not hold) the exact float64 mirror finds
// the reference's cell.  (The forward pass may
// settle a sample on value alone; the derivative needs the beamlet.)
__device__ int sample_beamlet(const BeamDev& b, const BeamletDev& bl, const GridDev& g, const float* pos,
                              const float* off, float rx, float ry, float rz, int ix, int iy, int iz, bool exact,
                              int& bad) {
  if (!b.geom_f32 && !exact) {
    const float p0 = pos[0] + rx, p1 = pos[1] + ry, p2 = pos[2] + rz;
    const float np_ = b.vyf[0] * p0 + b.vyf[1] * p1 + b.vyf[2] * p2;
    const float m0p = b.m0f[0] * p0 + b.m0f[1] * p1 + b.m0f[2] * p2;
    const float m2p = b.m2f[0] * p0 + b.m2f[1] * p1 + b.m2f[2] * p2;
    const float ndr = b.a_nS - np_;
    if (fabsf(ndr) > 0.2f * fabsf(b.a_K)) {
      const float si = __fdividef(b.a_K, ndr);
      const float ux = (b.a_c0 + si * (b.a_m0S - m0p)) * 100.0f;
      const float uz = (b.a_c2 + si * (b.a_m2S - m2p)) * 100.0f;
      const int i0 = floor_cell(ux - SAMPLE_DELTA), i1 = floor_cell(ux + SAMPLE_DELTA);
      const int k0 = floor_cell(uz - SAMPLE_DELTA), k1 = floor_cell(uz + SAMPLE_DELTA);
      const int id = beamlet_of(b, bl, i0, k0);
      if ((i0 == i1 && k0 == k1) ||
          (beamlet_of(b, bl, i1, k0) == id && beamlet_of(b, bl, i0, k1) == id && beamlet_of(b, bl, i1, k1) == id))
        return id;
    }
  }
  int fi, fk;
  if (!sample_cell_exact(b, g, pos, off, ix, iy, iz, bad, fi, fk)) return -1;
  return beamlet_of(b, bl, fi, fk);
}

// Row (or column) of beamlets of one sub-sample coordinate: v is its cell
// coordinate relative to the grid's first cell, n beamlets of `cell` cells.
// -1 outside the grid; within delta of an edge between beamlets or of the
// grid sets amb.
__device__ __forceinline__ int beamlet_index(float v, float cell, float inv_cell, int n, float delta, bool& amb) {
  const float q = floorf(v * inv_cell), d = v - q * cell;
  const bool in = q >= 0.0f && q < (float)n;
  amb = amb || ((d < delta || d > cell - delta) && q >= -1.0f && q <= (float)n);
  return in ? (int)q : -1;
}

// dL/dw for blocked(v) = sum_s w[beamlet(s)] / S^3 and T = blocked^2 * H
// (fluence and TERMA each carry one factor of blocked): over the voxels of
// the prologue's list with T != 0, g(v) = tbar(v) * 2 T(v) / blocked(v) is
// spread over the beamlets of its S^3 sub-samples, in float64.
//
// One voxel per lane, 32 consecutive entries of the list per warp.  With 3
// samples per axis and a shadow on at most 2 x 2 beamlets (a, c) .. (a + 1,
// c + 1), the samples in each are popcounts of two side tests (below_edge), and
// blocked is the counts' mean of the crop's values there.  Runs of lanes with
// the same beamlet (neighbours along z) are summed first, as float32 pairs, and
// add once, to L2: a histogram in shared memory adds float64 by compare-and-swap
// loops that the SM's warps, all at the same few beamlets, make each other
// repeat, and its flush costs as many global adds as this.  Other voxels go
// sample by sample and add per change of beamlet.
//
// 40 x 40 beamlets of 0.5 cm on 128^3 (one million voxels): one warp-wide sum
// per distinct beamlet 988 us (a line of 32 voxels crosses 16 of them; 128
// registers, one CTA per SM), runs into a shared histogram 420 us, into L2 390 us,
// with ambiguous samples decided one by one instead of the whole voxel 167 us.
constexpr int ADJ_THREADS = 256;
__global__ void __launch_bounds__(ADJ_THREADS, 3) blocked_adjoint_kernel(const __grid_constant__ GridDev g,
                                                                         const __grid_constant__ BeamDev b,
                                                                         const BeamletDev bl, int S,
                                                                         const float* __restrict__ T,
                                                                         const float* __restrict__ tbar,
                                                                         const int* __restrict__ list_count,
                                                                         const int* __restrict__ list_v,
                                                                         double* __restrict__ wbar,
                                                                         int* __restrict__ flags) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int count = *list_count;
  int bad = 0;
  float off[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) off[k] = fdiv(g.spacing[k], (float)S);
  const float cr = (float)bl.cell_rows, cc = (float)bl.cell_cols;
  const float icr = 1.0f / cr, icc = 1.0f / cc;
  // cell coordinate of the beamlet grid's first row and column
  const float u0 = (float)(bl.r0 - 1999), w0 = (float)(bl.c0 - 1999);
  // the grid ends where the map does: its last row and column are read by the wrapped index only
  const bool whole = bl.r0 + bl.rows * bl.cell_rows <= 3999 && bl.c0 + bl.cols * bl.cell_cols <= 3999;
  const unsigned stride = gridDim.x * blockDim.x, rounds = ((unsigned)count + stride - 1) / stride;
  for (unsigned it = 0; it < rounds; ++it) {
    const unsigned e = it * stride + blockIdx.x * blockDim.x + threadIdx.x;
    float t = 0.0f, tb = 0.0f, pos[3] = {0.0f, 0.0f, 0.0f};
    if (e < (unsigned)count) {
      const int v = list_v[e];
      const int z = v % g.n[2];
      const int r = v / g.n[2];
      const int y = r % g.n[1];
      const int x = r / g.n[1];
      t = T[((size_t)x * g.n[1] + y) * g.zp + z];
      tb = tbar[v];
      pos[0] = voxel_centre(g.origin[0], g.spacing[0], x);
      pos[1] = voxel_centre(g.origin[1], g.spacing[1], y);
      pos[2] = voxel_centre(g.origin[2], g.spacing[2], z);
    }
    unsigned cnt = 0;      // samples in beamlets (a, c), (a, c + 1), (a + 1, c), (a + 1, c + 1), a byte each
    int id0 = 0;           // beamlet (a, c), which may lie outside the grid
    float ghi = 0.0f, glo = 0.0f;   // g(v) / S^3
    if (t != 0.0f && tb != 0.0f) {
      Centre c;
      const bool lat = whole && lattice_centre(b, pos, c);
      bool done = false;
      if (lat && S == 3) {
        const int a = floor_int((c.u - c.mu - u0) * icr - 1e-3f), k = floor_int((c.w - c.mw - w0) * icc - 1e-3f);
        const float eu = u0 + (float)(a + 1) * cr, ew = w0 + (float)(k + 1) * cc;   // the lines between them
        if (c.u + c.mu < eu + cr && c.w + c.mw < ew + cc) {
          unsigned near = 0;
          unsigned in_u = c.u + c.mu < eu ? ALL_27 : below_edge(b, off, c, true, eu, 1.0f, near);
          unsigned in_w = c.w + c.mw < ew ? ALL_27 : below_edge(b, off, c, false, ew, 1.0f, near);
          for_mask(near, [&](unsigned bit, int ix, int iy, int iz) {
            int fi, fk;
            if (!sample_cell_exact(b, g, pos, off, ix, iy, iz, bad, fi, fk)) return;
            in_u = (float)fi < eu ? in_u | bit : in_u & ~bit;
            in_w = (float)fk < ew ? in_w | bit : in_w & ~bit;
          });
          done = true;
          id0 = a * bl.cols + k;
          double sum = 0.0;
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const int i = a + (f >> 1), j = k + (f & 1);
            if (i < 0 || i >= bl.rows || j < 0 || j >= bl.cols) continue;
            const int n = __popc(((f & 2) ? ~in_u & ALL_27 : in_u) & ((f & 1) ? ~in_w & ALL_27 : in_w));
            cnt |= (unsigned)n << (8 * f);
            if (n)
              sum = __fma_rn((double)n, (double)__ldg(b.block + (size_t)(i * bl.cell_rows) * b.bcols + j * bl.cell_cols),
                             sum);
          }
          // 2 t tb / S^3 / blocked with blocked = sum / S^3
          const double gv = sum > 0.0 ? 2.0 * (double)t * (double)tb / sum : 0.0;
          ghi = d2f(gv);
          glo = d2f(gv - (double)ghi);
        }
      }
      if (!done) {
        const double blocked = blocked_fraction<false>(b, g, S, pos, bad);
        const double gv = blocked > 0.0 ? (double)tb * 2.0 * (double)t / blocked / ((double)S * S * S) : 0.0;
        int cur = -1, n = 0;
        auto sample = [&](int id) {
          if (id == cur) {
            ++n;
          } else if (id >= 0) {
            if (n) atomicAdd(wbar + cur, gv * (double)n);
            cur = id;
            n = 1;
          }
        };
        if (gv == 0.0) {
        } else if (lat) {
          for_samples(b, off, S, c, [&](int ix, int iy, int iz, float u, float w) {
            bool amb = false;
            const int i = beamlet_index(u - u0, cr, icr, bl.rows, c.delta, amb);
            const int j = beamlet_index(w - w0, cc, icc, bl.cols, c.delta, amb);
            int id = (i < 0 || j < 0) ? -1 : i * bl.cols + j;
            if (amb) {
              int fi, fk;
              id = sample_cell_exact(b, g, pos, off, ix, iy, iz, bad, fi, fk) ? beamlet_of(b, bl, fi, fk) : -1;
            }
            sample(id);
          });
        } else {
          const bool exact = general_exact(b, pos);
          for (int ix = 0; ix < S; ++ix)
            for (int iy = 0; iy < S; ++iy)
              for (int iz = 0; iz < S; ++iz) {
                const float rx = off[0] * ((float)ix + 0.5f) - g.spacing[0] * 0.5f;
                const float ry = off[1] * ((float)iy + 0.5f) - g.spacing[1] * 0.5f;
                const float rz = off[2] * ((float)iz + 0.5f) - g.spacing[2] * 0.5f;
                sample(sample_beamlet(b, bl, g, pos, off, rx, ry, rz, ix, iy, iz, exact, bad));
              }
        }
        if (n) atomicAdd(wbar + cur, gv * (double)n);
      }
    }
    // byte fields: suffix sums over runs of lanes with the same beamlet, added by each run's first lane.
    // A lane without samples in a beamlet brings nothing to it, and a run without any adds nothing: the
    // beamlet may lie off the grid, and a share that is not finite (a NaN in the dose gradient) times a
    // count of 0 is not 0
    const int next_id = __shfl_down_sync(full, id0, 1);
    const unsigned same_next = __ballot_sync(full, lane < 31 && id0 == next_id);   // lane and lane + 1
    const int run = __clz(__brev(~(same_next >> lane)));           // lanes of the run after this one
    const bool first = lane == 0 || !((same_next >> (lane - 1)) & 1u);
#pragma unroll 1
    for (int f = 0; f < 4; ++f) {
      const float n = (float)((cnt >> (8 * f)) & 255u);
      const unsigned has = __ballot_sync(full, n > 0.0f);
      if (!has) continue;
      float hi = 0.0f, lo = 0.0f;
      if (n > 0.0f) {
        hi = ghi * n;
        lo = __fmaf_rn(ghi, n, -hi) + glo * n;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float h2 = __shfl_down_sync(full, hi, o), l2 = __shfl_down_sync(full, lo, o);
        if (o <= run) {
          const float t2 = fadd(hi, h2), bb = fsub(t2, hi);
          lo = fadd(fadd(lo, l2), fadd(fsub(hi, fsub(t2, bb)), fsub(h2, bb)));
          hi = t2;
        }
      }
      const double sum = fabsf(hi) <= 3.4028234e38f ? (double)hi + (double)lo : (double)hi;
      const bool any = ((has >> lane) & ((2u << run) - 1u)) != 0;    // in this lane or the run's after it
      if (first && any && sum != 0.0) atomicAdd(wbar + id0 + (f >> 1) * bl.cols + (f & 1), sum);
    }
  }
  if (__any_sync(full, bad) && lane == 0) atomicOr(flags, FLAG_PARALLEL_RAY);
}

cudaError_t launch_blocked_adjoint(const GridDev& g, const BeamDev& b, const BeamletDev& bl, int S, const float* T,
                                   const float* tbar, const int* list_count, const int* list_v, double* wbar,
                                   int n_sm, int* flags, cudaStream_t st) {
  blocked_adjoint_kernel<<<n_sm * 3, ADJ_THREADS, 0, st>>>(g, b, bl, S, T, tbar, list_count, list_v, wbar, flags);
  return cudaGetLastError();
}

void upload_unit_partials() {
  double p[28];
  p[0] = 0.0;
  const double q = 1.0 / 27.0;
  for (int i = 1; i < 28; ++i) p[i] = p[i - 1] + q;
  cudaMemcpyToSymbol(c_unit_partial, p, sizeof(p));
  double full[17] = {0.0}, inv[17] = {0.0};
  for (int S = 1; S <= 16; ++S) {
    inv[S] = 1.0 / (double)(S * S * S);
    for (int i = 0; i < S * S * S; ++i) full[S] += inv[S];
  }
  cudaMemcpyToSymbol(c_inv_count, inv, sizeof(inv));
  cudaMemcpyToSymbol(c_unit_sum, full, sizeof(full));
}

void launch_prologue(const float* rho, const GridDev& g, const BeamDev& b, const SettingsDev& s, float* T,
                     const Inter& inter, int all_voxels, int* aabb, bool box, int* list_v, int n_sm, int* flags,
                     cudaStream_t st, int ctas_per_sm) {
  const long long N = (long long)g.n[0] * g.n[1] * g.n[2];
  const int threads = 256;
  const long long lines = (long long)g.n[0] * g.n[1];
  int* list_count = aabb + 6;
  // without a list (all voxels) the TERMA pass takes them in order and writes
  // every one: there is nothing to cull or to zero (96^3 with every
  // intermediate: 20 of 209 us)
  if (list_v)
    cull_kernel<<<(unsigned)((lines + 7) / 8), threads, 0, st>>>(g, b, T, inter, all_voxels, list_count, list_v);
  const long long want = (N + threads - 1) / threads;
  const long long cap = (long long)n_sm * ctas_per_sm;
  const int grid = (int)(want < cap ? want : cap);
  terma_kernel<<<grid > 0 ? grid : 1, threads, 0, st>>>(rho, g, b, s, T, inter, all_voxels, list_count, list_v,
                                                        box ? aabb : nullptr, flags);
}

// Batched prologue (no intermediates): one cull launch over every beam's grid
// and one TERMA launch whose warps claim chunks of every beam's list from one
// counter, so all beams run together and no beam leaves a tail.
void launch_prologue_batch(const PrologueBeam* recs, int n_beams, long long max_voxels, long long max_lines,
                           int n_sm, int* flags, int* work, cudaStream_t st, int ctas_per_sm) {
  const int threads = 256;
  // lines per warp: enough warps for every SM's resident ones, at most 32 lines
  int lpw = 4;
  while (lpw < 32 && max_lines * n_beams > (long long)n_sm * 64 * lpw) lpw *= 2;
  const long long per = lpw * (threads / 32);
  launch_after(true, cull_batch_kernel, dim3((unsigned)((max_lines + per - 1) / per), n_beams), threads, 0, st, recs, lpw);
  // persistent: at most the resident CTAs (3 per SM at 80 registers), fewer
  // for small batches; the warps share all beams' chunks
  const long long want = ((long long)n_beams * max_voxels + threads - 1) / threads;
  const long long cap = (long long)n_sm * std::min(ctas_per_sm, 3);
  launch_after(true, terma_batch_kernel, dim3((unsigned)std::max(1ll, std::min(cap, want))), threads, 0, st, recs, n_beams,
               flags, work);
}

__global__ void init_scratch_kernel(int* aabb, int n_beams, int* counters, unsigned keep) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  // per beam: lo/hi pairs of the TERMA box, then the prologue list count
  if (i < n_beams * 8) aabb[i] = (i % 8 >= 6) ? 0 : ((i % 2 == 0) ? INT_MAX : INT_MIN);
  if (i < 8 && !((keep >> i) & 1u)) counters[i] = 0;
}

void launch_init_scratch(int* aabb, int n_beams, int* counters, cudaStream_t st, unsigned keep) {
  const int n = n_beams * 8 > 8 ? n_beams * 8 : 8;
  init_scratch_kernel<<<(n + 255) / 256, 256, 0, st>>>(aabb, n_beams, counters, keep);
}

}  // namespace ch
