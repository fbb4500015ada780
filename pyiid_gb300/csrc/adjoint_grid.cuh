// adjoint_grid.cuh -- the position gradient of Rw or chi^2 from a table of
// the pair force.
//
// As in debye_kernels.cuh (get_grad_rw / get_grad_chi_sq, pyiid/experiments/
// elasticscatter/kernels/master_kernel.py:293-376, moved back to the bins):
//   d(potential)/dx_a = sum_b (x_a - x_b) s_ab,
//   s_ab = sum_k W_k (Q_k cos(Q_k r) - sin(Q_k r)/r) / r^2
// with W_k one number per bin, configuration and species pair.  So with
//   B(u) = sum_k W_k sin(k theta),  theta = dq r = 2 pi u / M,
// s_ab = (c B'(u) - B(u)/r) / r^2 with c = du/dr: one function of one
// variable for all pairs of a key.  adjoint_grid_table_kernel tabulates it,
// adjoint_grid_kernel reads it once per unordered pair.
#pragma once

#include "debye_kernels.cuh"
#include "phase_grid.cuh"

namespace pyiid {

// Cells per period: 8 per bin.  A cell then spans k (2 pi / M) <= pi/4 of
// phase, and a polynomial of degree 7 about its centre, |t| <= 1/2, holds
// the sine to 1e-10 and the derivative to 2e-8 of sum |k W_k| (t^8, the
// first term left out of the cosine's series, is replaced by the
// lower-degree polynomial nearest to it).  Finer cells would shorten the
// polynomial by one term per halving and double the table; at 330 bins a
// key's table takes 42 KB of shared memory, four CTAs per SM.
constexpr int kAdjCellsPerBin = 8;
constexpr int kAdjCoef = 8;     // polynomial coefficients per cell
constexpr int kAdjBlock = 256;  // threads of both kernels

// wk[key][k][p]: W_k times the coefficient of t^p in cos(k delta t) (p even)
// and sin(k delta t) (p odd), delta = 2 pi / M; zero below kmin or where
// na_k = 0.  key = configuration x species pair (sa >= sb).
struct WkArgs {
  const double *na;
  const float *ftab;
  const int2 *spair_species;
  int n_spairs;
  float delta;
  float4 *wk;
};

// the weights of configuration b and bin k from w_k
__device__ __forceinline__ void adjoint_grid_weights(const WkArgs &a, int b,
                                                     int k, bool on, int n_bins,
                                                     double w) {
  const double nak = a.na[(size_t)b * n_bins + k];
  const double w2 = on && nak != 0.0 ? 2.0 * w / nak : 0.0;
  // Taylor terms z^p / p! of z = k delta <= pi/4; with tau = 2 t,
  // tau^8 = 2 tau^6 - 5/4 tau^4 + tau^2/4 - 1/128 + T_8(tau)/128
  const float z = (float)k * a.delta, z2 = z * z;
  const float z4 = z2 * z2;
  const float e8 = z4 * z4 * (1.0f / 40320.0f);
  const float e0 = 1.0f - e8 * (1.0f / 32768.0f);
  const float e2 = -0.5f * z2 + e8 * (1.0f / 256.0f);
  const float e4 = z4 * (1.0f / 24.0f) - e8 * (5.0f / 64.0f);
  const float e6 = -z4 * z2 * (1.0f / 720.0f) + e8 * 0.5f;
  const float o3 = -z * z2 * (1.0f / 6.0f), o5 = z * z4 * (1.0f / 120.0f);
  const float o7 = -z * z4 * z2 * (1.0f / 5040.0f);
  for (int s = 0; s < a.n_spairs; ++s) {
    const int2 ss = a.spair_species[s];
    const float W = (float)(w2 * (double)a.ftab[ss.x * n_bins + k] *
                            (double)a.ftab[ss.y * n_bins + k]);
    float4 *o = a.wk + 2 * (((size_t)b * a.n_spairs + s) * n_bins + k);
    o[0] = make_float4(W * e0, W * z, W * e2, W * o3);
    o[1] = make_float4(W * e4, W * o5, W * e6, W * o7);
  }
}

// tab[key][j][p], cell centres u = j, 0 <= j <= M/2 (B is odd in u, so half
// a period is enough): even p sum wk sin(k theta_j), odd p sum wk
// cos(k theta_j).  The cell j' = M/2 - j has sin(k theta_j') = -(-1)^k
// sin(k theta_j) and cos(k theta_j') = (-1)^k cos(k theta_j), so the sums of
// even and of odd bins, kept apart, give both cells for one.
// Lane = cell j <= M/4, the eight warps each take an eighth of every chunk of
// bins (keeps the chains of FP32 additions short: 42 bins at 330) and are
// added in a fixed order.  Bins go in blocks of eight around an accurate
// centre, each one rotation by +-n theta_j, n <= 4, away from it, so no error
// builds up along k.  What bounds it is the reads of wk (two of 16 bytes per
// bin and warp, four cycles each): 38 us for 64 keys of 330 bins with one
// cell per lane, 20 with two.
constexpr int kAdjChunk = 512;  // bins staged in shared memory (16 KB)
__global__ void __launch_bounds__(kAdjBlock)
    adjoint_grid_table_kernel(const float4 *__restrict__ wk, int n_bins,
                              int kmin, int m, float inv_m,
                              float4 *__restrict__ tab) {
  __shared__ float4 sw[2 * kAdjChunk];
  __shared__ float red[8][kAdjCoef][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_cells = m / 2 + 1, n_half = m / 4 + 1;
  const int j = min((int)(blockIdx.x * 32 + lane), n_half - 1);
  const size_t key = blockIdx.y;
  float sn[4], cn[4];
#pragma unroll
  for (int n = 0; n < 4; ++n)
    sincos_turn((n + 1) * j % m, m, inv_m, sn[n], cn[n]);
  float acc[2][kAdjCoef];  // even, odd bins
#pragma unroll
  for (int p = 0; p < kAdjCoef; ++p) acc[0][p] = acc[1][p] = 0.f;
  for (int k0 = kmin & ~1; k0 < n_bins; k0 += kAdjChunk) {
    const int nb = min(kAdjChunk, n_bins - k0);
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * kAdjChunk; i += kAdjBlock)
      sw[i] = i < 2 * nb ? wk[2 * (key * n_bins + k0) + i]
                         : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    const int per = ((nb + 7) / 8 + 7) / 8 * 8;  // bins per warp
    const int i1 = min((warp + 1) * per, nb);
    for (int i0 = warp * per; i0 < i1; i0 += 8) {
      // (12,292 x 24,577 stays under 2^31)
      float sc, cc;
      sincos_turn((k0 + i0 + 4) * j % m, m, inv_m, sc, cc);
#pragma unroll
      for (int n = -4; n < 4; ++n) {
        const int i = i0 + 4 + n;  // < 512; weights past nb are zero
        float s = sc, c = cc;
        if (n > 0) {
          s = fmaf(cc, sn[n - 1], sc * cn[n - 1]);
          c = fmaf(-sc, sn[n - 1], cc * cn[n - 1]);
        } else if (n < 0) {
          s = fmaf(-cc, sn[-n - 1], sc * cn[-n - 1]);
          c = fmaf(sc, sn[-n - 1], cc * cn[-n - 1]);
        }
        float(&part)[kAdjCoef] = acc[n & 1];
        const float4 a = sw[2 * i], b = sw[2 * i + 1];
        part[0] = fmaf(a.x, s, part[0]);
        part[1] = fmaf(a.y, c, part[1]);
        part[2] = fmaf(a.z, s, part[2]);
        part[3] = fmaf(a.w, c, part[3]);
        part[4] = fmaf(b.x, s, part[4]);
        part[5] = fmaf(b.y, c, part[5]);
        part[6] = fmaf(b.z, s, part[6]);
        part[7] = fmaf(b.w, c, part[7]);
      }
    }
  }
  // thread = (cell, coefficient): the eight warps' sums, pairwise; even bins
  // first, then odd ones
  const int cell = threadIdx.x >> 3, p = threadIdx.x & 7;
  float sum[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kAdjCoef; ++q) red[warp][q][lane] = acc[e][q];
    __syncthreads();
    sum[e] = ((red[0][p][cell] + red[1][p][cell]) +
              (red[2][p][cell] + red[3][p][cell])) +
             ((red[4][p][cell] + red[5][p][cell]) +
              (red[6][p][cell] + red[7][p][cell]));
  }
  const int jj = blockIdx.x * 32 + cell;
  if (jj >= n_half) return;
  float *out = reinterpret_cast<float *>(tab) + key * n_cells * kAdjCoef + p;
  // (even p: sines, odd p: cosines; the middle cell is its own image)
  out[(size_t)jj * kAdjCoef] = sum[0] + sum[1];
  if (2 * jj < n_cells - 1)
    out[(size_t)(n_cells - 1 - jj) * kAdjCoef] =
        (p & 1) ? sum[0] - sum[1] : sum[1] - sum[0];
}

// grad[a] = sum_b s_ab (x_a - x_b), each unordered pair once.  CTA = work item
// (tile I, a run of tiles J <= I of one species); a warp takes a tile J, or a
// share of the 32 steps of one where the run is shorter than five.  Lane a
// holds atom a of I and in step s meets atom (a + s) mod 32 of J; the force
// on that atom is summed in a register that moves one lane down per step, so
// it stays with its atom (three shuffles a step; a warp sum would take
// fifteen).  Atoms of one tile meet in all 31 ordered steps instead.  The
// partial rows of I and J go to part (as adjoint_sym_kernel's) and
// adjoint_reduce_kernel adds them in a fixed order.
// Bound by the shared-memory pipe: the two 16-byte reads of the table at 32
// unrelated cells take about ten cycles each.  They come from two planes: one
// of 32-byte cells has only every second bank group at a time and took 14.
// TAB_SMEM: the key's table is staged in shared memory; else it is read
// through L1 (it does not fit for more than about 850 bins, and an item of one
// tile pair does not earn the copy).  A pair at r = 0 gives NaN, as the closed
// form does.
// 64 x 1,000 atoms, 330 bins: 173 us and 9 for the reduction, after 20 us for
// the tables (adjoint_sym_kernel and its reduction: 2,470 us; with each
// ordered pair evaluated 244); the gradient is 1.1e-7 off the FP64 one
// (2.3e-7).
template <bool TAB_SMEM>
__global__ void __launch_bounds__(kAdjBlock)
    adjoint_grid_kernel(const float *__restrict__ pos,
                        const int *__restrict__ perm,
                        const int4 *__restrict__ tiles,
                        const int4 *__restrict__ items,
                        const int *__restrict__ order, GridScale gs,
                        int n_cells, const float4 *__restrict__ tab,
                        const int *__restrict__ ioff,
                        const int *__restrict__ joff, float *__restrict__ part) {
  extern __shared__ float4 stab[];  // [2][n_cells]
  constexpr int W = kAdjBlock / 32;
  __shared__ float4 sJ[W][kTile][2];  // (hx, hy, hz, lx), (ly, lz, 0, 0)
  __shared__ float sred[W][kTile][3];
  __shared__ float sjac[W][kTile][3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int item = order[blockIdx.x];
  const int4 it = items[item];
  const int4 ti = tiles[it.x];
  const int len = it.z - it.y;
  const float4 *src = tab + (size_t)it.w * n_cells * 2;
  if (TAB_SMEM)
    for (int i = threadIdx.x; i < 2 * n_cells; i += kAdjBlock)
      stab[(i & 1) * n_cells + (i >> 1)] = src[i];
  const bool here = lane < ti.y;
  const float4 pa = load_atom(pos, perm, ti.x + min(lane, ti.y - 1));
  SplitAtom a = split_atom(pa.x, pa.y, pa.z);
  if (!here) a.hx += 1.0f;  // counts nothing; any place of its own
  if (TAB_SMEM) __syncthreads();
  // tasks: (tile of the run, share of its steps)
  const int shares = len > 4 ? 1 : len > 2 ? 2 : len == 2 ? 4 : 8;
  const int per = kTile / shares;
  float *const pj = part + joff[item];
  float gx = 0.f, gy = 0.f, gz = 0.f;
  for (int task = warp; task < len * shares; task += W) {
    const int jl = task / shares, tj = it.y + jl;
    const int4 tJ = tiles[tj];
    const bool diag = tj == it.x;
    const float4 q = load_atom(pos, perm, tJ.x + min(lane, tJ.y - 1));
    SplitAtom mine = split_atom(q.x, q.y, q.z);
    if (lane >= tJ.y) mine.hx += 2.0f;
    __syncwarp();
    sJ[warp][lane][0] = make_float4(mine.hx, mine.hy, mine.hz, mine.lx);
    sJ[warp][lane][1] = make_float4(mine.ly, mine.lz, 0.f, 0.f);
    __syncwarp();
    const int s0 = (task % shares) * per, s1 = s0 + per;
    float jx = 0.f, jy = 0.f, jz = 0.f;
#pragma unroll 2
    for (int s = s0; s < s1; ++s) {
      const int bl = (lane + s) & (kTile - 1);
      const float4 q0 = sJ[warp][bl][0];
      const float2 q1 = *reinterpret_cast<const float2 *>(&sJ[warp][bl][1]);
      SplitAtom b{q0.x, q0.y, q0.z, q0.w, q1.x, q1.y};
      const bool self = diag && s == 0;
      if (self) b.hx += 1.0f;  // any distance but 0
      const PairDist p = pair_dist(a, b);
      float uh, ul;
      grid_pos(gs, p.r, p.rl, uh, ul);
      const float sg = uh < 0.f ? -1.0f : 1.0f;
      uh *= sg;
      ul *= sg;
      const float fj = rintf(uh);
      const float t = (uh - fj) + ul;
      const int j = min(max((int)fj, 0), n_cells - 1);
      const float4 lo4 = TAB_SMEM ? stab[j] : src[2 * j];
      const float4 hi4 = TAB_SMEM ? stab[n_cells + j] : src[2 * j + 1];
      // value and derivative together
      float v = hi4.w, d = hi4.w;
      v = fmaf(v, t, hi4.z);
      d = fmaf(d, t, v);
      v = fmaf(v, t, hi4.y);
      d = fmaf(d, t, v);
      v = fmaf(v, t, hi4.x);
      d = fmaf(d, t, v);
      v = fmaf(v, t, lo4.w);
      d = fmaf(d, t, v);
      v = fmaf(v, t, lo4.z);
      d = fmaf(d, t, v);
      v = fmaf(v, t, lo4.y);
      d = fmaf(d, t, v);
      v = fmaf(v, t, lo4.x);
      float f = fmaf(gs.hi, d, -(sg * v) * p.inv_r) * (p.inv_r * p.inv_r);
      if (!here || bl >= tJ.y || self) f = 0.f;
      gx = fmaf(f, p.dx, gx);
      gy = fmaf(f, p.dy, gy);
      gz = fmaf(f, p.dz, gz);
      jx = fmaf(-f, p.dx, jx);
      jy = fmaf(-f, p.dy, jy);
      jz = fmaf(-f, p.dz, jz);
      if (s + 1 < s1) {
        const int from = (lane + 1) & (kTile - 1);
        jx = __shfl_sync(0xffffffffu, jx, from);
        jy = __shfl_sync(0xffffffffu, jy, from);
        jz = __shfl_sync(0xffffffffu, jz, from);
      }
    }
    // (in its own tile every atom has its row on the i side already)
    if (diag) jx = jy = jz = 0.f;
    const int bl = (lane + s1 - 1) & (kTile - 1);
    float *o = shares == 1 ? pj + (size_t)jl * kTile * 3 : &sjac[task][0][0];
    o[bl * 3] = jx;
    o[bl * 3 + 1] = jy;
    o[bl * 3 + 2] = jz;
  }
  // (an atom against itself counts nothing, whatever its place: 0 x NaN)
  if (ti.y == 1 && it.y == it.x) gx = gy = gz = 0.f;
  sred[warp][lane][0] = gx;
  sred[warp][lane][1] = gy;
  sred[warp][lane][2] = gz;
  __syncthreads();
  float *pi = part + ioff[item];
  for (int i = threadIdx.x; i < kTile * 3; i += kAdjBlock) {
    float sum = 0.f;
    for (int g = 0; g < W; ++g) sum += (&sred[g][0][0])[i];
    pi[i] = sum;
  }
  if (shares > 1)
    for (int i = threadIdx.x; i < len * kTile * 3; i += kAdjBlock) {
      const int jl = i / (kTile * 3), c = i % (kTile * 3);
      float sum = 0.f;
      for (int g = 0; g < shares; ++g)
        sum += (&sjac[jl * shares + g][0][0])[c];
      pj[i] = sum;
    }
}

}  // namespace pyiid
