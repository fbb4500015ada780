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
// adjoint_grid_kernel reads it once per ordered pair.
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

// grad[a] = sum_b s_ab (x_a - x_b).  CTA = tile I, lane = atom a of it; the
// eight warps share the atoms b, staged kAdjBlock at a time, so all lanes of
// a warp read one b (a broadcast) and the table at 32 unrelated cells.  Each
// ordered pair is evaluated: the unordered half would save the distance of
// every second pair but need its force carried to the other atom (six
// shuffles and a second pass over partial rows).  About 75 instructions per
// 32 pairs; the two 16-byte table reads, 8 to 10 shared-memory cycles each,
// run beside them.  TAB_SMEM: the key's table is staged in shared memory
// (it does not fit for more than about 850 bins: then it is read through
// L1).  A pair at r = 0 gives NaN, as the closed form does.
// 64 x 1,000 atoms, 330 bins: 244 us, after 20 us for the tables
// (adjoint_sym_kernel and its reduction: 2,470 us); the gradient
// is 1.1e-7 off the FP64 one (2.3e-7).
template <bool TAB_SMEM>
__global__ void __launch_bounds__(kAdjBlock)
    adjoint_grid_kernel(const float *__restrict__ pos,
                        const int *__restrict__ perm,
                        const int4 *__restrict__ tiles,
                        const int2 *__restrict__ cfg_tiles, GridScale gs,
                        int n_cells, const float4 *__restrict__ tab,
                        int n_spairs, float *__restrict__ grad) {
  extern __shared__ float4 stab[];
  __shared__ float4 sB[2][kAdjBlock];  // (hx, hy, hz, lx), (ly, lz, 0, 0)
  __shared__ float sred[kAdjBlock / kTile][kTile][3];
  const int4 ti = tiles[blockIdx.x];
  const int2 ct = cfg_tiles[ti.z];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ia = ti.x + min(lane, ti.y - 1);  // sorted index of this atom
  const float4 pa = load_atom(pos, perm, ia);
  const SplitAtom a = split_atom(pa.x, pa.y, pa.z);
  float gx = 0.f, gy = 0.f, gz = 0.f;
  for (int tj = ct.x; tj < ct.y;) {
    // the run of tiles of one species: atoms [b0, b1) in sorted order
    const int sb = tiles[tj].w, b0 = tiles[tj].x;
    int b1 = b0;
    for (; tj < ct.y && tiles[tj].w == sb; ++tj) b1 += tiles[tj].y;
    const int hi = max(ti.w, sb), lo = min(ti.w, sb);
    const size_t key = (size_t)ti.z * n_spairs + hi * (hi + 1) / 2 + lo;
    const float4 *src = tab + key * n_cells * 2;
    __syncthreads();
    if (TAB_SMEM)
      for (int i = threadIdx.x; i < 2 * n_cells; i += kAdjBlock)
        stab[i] = src[i];
    for (int c0 = b0; c0 < b1; c0 += kAdjBlock) {
      const int nb = min(kAdjBlock, b1 - c0);
      __syncthreads();
      if ((int)threadIdx.x < nb) {
        const float4 q = load_atom(pos, perm, c0 + threadIdx.x);
        const SplitAtom s = split_atom(q.x, q.y, q.z);
        sB[0][threadIdx.x] = make_float4(s.hx, s.hy, s.hz, s.lx);
        sB[1][threadIdx.x] = make_float4(s.ly, s.lz, 0.f, 0.f);
      }
      __syncthreads();
      auto sweep = [&](auto checked) {
        constexpr bool CHECK = decltype(checked)::value;
#pragma unroll 2
        for (int i = warp; i < nb; i += kAdjBlock / 32) {
          const bool self = CHECK && c0 + i == ia;
          const float4 q0 = sB[0][i];
          const float2 q1 = *reinterpret_cast<const float2 *>(&sB[1][i]);
          SplitAtom b{q0.x, q0.y, q0.z, q0.w, q1.x, q1.y};
          if (CHECK && self) b.hx += 1.0f;  // any distance but 0
          const PairDist p = pair_dist(a, b);
          float uh, ul;
          grid_pos(gs, p.r, p.rl, uh, ul);
          const float sg = uh < 0.f ? -1.0f : 1.0f;
          uh *= sg;
          ul *= sg;
          const float fj = rintf(uh);
          const float t = (uh - fj) + ul;
          const int j = min(max((int)fj, 0), n_cells - 1);
          const float4 *cp = TAB_SMEM ? stab + 2 * j : src + 2 * j;
          const float4 lo4 = cp[0], hi4 = cp[1];
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
          float s = fmaf(gs.hi, d, -(sg * v) * p.inv_r) *
                    (p.inv_r * p.inv_r);
          if (CHECK && self) s = 0.f;
          gx = fmaf(s, p.dx, gx);
          gy = fmaf(s, p.dy, gy);
          gz = fmaf(s, p.dz, gz);
        }
      };
      if (c0 < ti.x + ti.y && ti.x < c0 + nb)
        sweep(BoolTag<true>());
      else
        sweep(BoolTag<false>());
    }
  }
  sred[warp][lane][0] = gx;
  sred[warp][lane][1] = gy;
  sred[warp][lane][2] = gz;
  __syncthreads();
  if ((int)threadIdx.x < ti.y * 3) {
    const int al = threadIdx.x / 3, c = threadIdx.x % 3;
    float sum = 0.f;
    for (int g = 0; g < kAdjBlock / kTile; ++g) sum += sred[g][al][c];
    grad[(size_t)perm[ti.x + al] * 3 + c] = sum;
  }
}

}  // namespace pyiid
