// phase_grid.cuh -- pair distances for the kernels that work on a grid of
// phases instead of on (pair, bin) terms.
//
// The bins Q_k = k dq are uniform, so every Debye quantity of a pair depends
// on its distance alone and is a trigonometric polynomial of degree < K in
// theta = dq r, of period 2 pi.  The kernels built on this header therefore
// lay a grid of M cells over one period, u = theta M / (2 pi), and take what
// a pair needs from (or add what it gives to) the few cells around its u.
// A pair then costs about a hundred instructions whatever the number of
// bins, where the recurrences of pair_math.cuh cost 1.5 to 8.5 lane
// operations per bin.
#pragma once

#include <cuda_runtime.h>

#include "pair_math.cuh"

namespace pyiid {

// u = r * scale for a grid of M cells per period of theta = dq r
struct GridScale {
  float hi, lo;   // M dq / (2 pi) as a float pair
  float m, inv_m; // M and 1 / M
};

// A coordinate split on the grid of 1/32: x = h + l exactly, |l| <= 1/64.
__device__ __forceinline__ void split_coord(float x, float &h, float &l) {
  h = rintf(x * 32.0f) * 0.03125f;
  l = __fsub_rn(x, h);
}

struct SplitAtom {
  float hx, hy, hz, lx, ly, lz;
};

__device__ __forceinline__ SplitAtom split_atom(float x, float y, float z) {
  SplitAtom s;
  split_coord(x, s.hx, s.lx);
  split_coord(y, s.hy, s.ly);
  split_coord(z, s.hz, s.lz);
  return s;
}

struct PairDist {
  float dx, dy, dz;  // x_a - x_b
  float r, rl;       // |x_a - x_b| as a float pair
  float inv_r;
};

// The general form: every difference and square as an error-free pair.
static __device__ __noinline__ PairDist pair_dist_general(float ax, float ay,
                                                          float az, float bx,
                                                          float by, float bz) {
  PairDist p;
  float xl, yl, zl;
  two_sum(ax, -bx, p.dx, xl);
  two_sum(ay, -by, p.dy, yl);
  two_sum(az, -bz, p.dz, zl);
  float s0, e0, s1, e1, s2, e2;
  two_prod(p.dx, p.dx, s0, e0);
  two_prod(p.dy, p.dy, s1, e1);
  two_prod(p.dz, p.dz, s2, e2);
  float h, l, h2, l2;
  two_sum(s0, s1, h, l);
  two_sum(h, s2, h2, l2);
  const float lo =
      l + l2 + e0 + e1 + e2 + 2.0f * (p.dx * xl + p.dy * yl + p.dz * zl);
  float r2h, r2l;
  fast_two_sum(h2, lo, r2h, r2l);
  p.r = __fsqrt_rn(r2h);
  const float res = __fmaf_rn(-p.r, p.r, r2h);
  p.inv_r = __frcp_rn(p.r);
  p.rl = __fmul_rn(__fadd_rn(res, r2l), 0.5f * p.inv_r);
  return p;
}

// |x_a - x_b| as a float pair.  The differences of the 1/32 parts are exact,
// and so is the sum n of their squares up to 128 A (24 bits); what the rest
// adds, c = sum dl (2 dh + dl), carries an absolute error of 2^-24 c, which
// is under 1e-8 A in r.  That is half the operations of the error-free form
// (27 against 58).  False for pairs nearer than 0.1 A or further than 128 A,
// where the argument fails, and for NaN: they take the general form.
__device__ __forceinline__ bool pair_dist_fast(const SplitAtom &a,
                                               const SplitAtom &b,
                                               PairDist &p) {
  const float hx = a.hx - b.hx, hy = a.hy - b.hy, hz = a.hz - b.hz;
  const float lx = a.lx - b.lx, ly = a.ly - b.ly, lz = a.lz - b.lz;
  const float n = fmaf(hx, hx, fmaf(hy, hy, hz * hz));
  const float c = fmaf(lx, fmaf(2.0f, hx, lx),
                       fmaf(ly, fmaf(2.0f, hy, ly), lz * fmaf(2.0f, hz, lz)));
  const float s = __fadd_rn(n, c);
  const float e = __fadd_rn(__fsub_rn(n, s), c);
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
  const float r = __fmul_rn(s, y);
  const float hy2 = 0.5f * y;
  p.r = r;
  p.rl = __fmul_rn(hy2, __fadd_rn(__fmaf_rn(-r, r, s), e));
  p.inv_r = fmaf(hy2, __fmaf_rn(-r, y, 1.0f), y);
  p.dx = hx + lx;
  p.dy = hy + ly;
  p.dz = hz + lz;
  return s > 0.01f && n < 16384.0f;
}

__device__ __forceinline__ PairDist pair_dist_general(const SplitAtom &a,
                                                      const SplitAtom &b) {
  return pair_dist_general(a.hx + a.lx, a.hy + a.ly, a.hz + a.lz, b.hx + b.lx,
                           b.hy + b.ly, b.hz + b.lz);
}

__device__ __forceinline__ PairDist pair_dist(const SplitAtom &a,
                                              const SplitAtom &b) {
  PairDist p;
  if (!pair_dist_fast(a, b, p)) p = pair_dist_general(a, b);
  return p;
}

// Grid position of a distance: u = r scale as a float pair (uh, ul), taken
// to [-M/2, M/2] by n whole periods (the multiple of M is exact); returns n.
__device__ __forceinline__ float grid_pos(const GridScale &g, float r,
                                          float rl, float &uh, float &ul) {
  float p, e;
  two_prod(g.hi, r, p, e);
  ul = fmaf(g.hi, rl, fmaf(g.lo, r, e));
  const float n = rintf(p * g.inv_m);
  uh = __fmaf_rn(-n, g.m, p);
  return n;
}

// sin and cos of 2 pi i / m for 0 <= i < m: the fraction 2 i / m is rounded
// once and the rounding, exact from one FMA, goes in by the derivative.
__device__ __forceinline__ void sincos_turn(int i, int m, float inv_m, float &s,
                                            float &c) {
  const int i2 = 2 * i > m ? 2 * i - 2 * m : 2 * i;
  const float a = (float)i2, fm = (float)m;
  const float x = a * inv_m;
  const float d = 3.14159265f * (__fmaf_rn(-x, fm, a) * inv_m);
  float s0, c0;
  sincospif(x, &s0, &c0);
  s = fmaf(c0, d, s0);
  c = fmaf(-s0, d, c0);
}

}  // namespace pyiid
