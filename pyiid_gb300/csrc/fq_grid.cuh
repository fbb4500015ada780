// fq_grid.cuh -- F(Q) of a configuration by spreading its pairs on a phase
// grid.
//
// sum over pairs of sin(Q_k r)/r (cpu_flat.py:79-114, gpu_flat.py:73-112 of
// pyiid/experiments/elasticscatter/kernels) is a sine transform of weights
// 1/r at the points u = r M dq / (2 pi) of a period of M cells.  Every pair
// is spread on its eight nearest cells with a Kaiser-Bessel window phi,
//   H_j = sum_pairs phi(j - u) / r,
// and the sums follow from one transform per (configuration, species pair),
//   D_k = (1 / phihat_k) sum_j H_j sin(2 pi k j / M),
// the usual non-uniform transform (Kaiser-Bessel gridding; Fessler and
// Sutton, IEEE Trans. Signal Process. 51, 2003).  What is left out is the
// window's spectrum beyond the period: 2e-8 rms of a term at M = 5 n_bins,
// against 2e-7 for the seeds and the recurrence of the direct kernels.
#pragma once

#include "debye_kernels.cuh"
#include "phase_grid.cuh"

namespace pyiid {

constexpr int kTaps = 8;        // cells a pair is spread on
constexpr int kTapCoef = 8;     // polynomial coefficients of a tap
constexpr int kFqCellsPerBin = 5;
constexpr int kNearTerms = 5;   // power sums of pairs at tiny distances
constexpr float kNearPhase = 0.6f;  // ... with Q_max r below this

// A histogram in memory: 8 words of power sums, then cells -3 .. used + 4.
constexpr int kGridCell0 = 8 + 3;  // word of cell 0
__host__ __device__ constexpr int grid_words(int used) {
  return kGridCell0 + used + 5;
}

// One row of work: tile I (atoms [a0, a0 + na) in sorted order) against the
// atoms [b0, b0 + nb) of one species; only b < a counts.  key: rank of the
// (configuration, species pair) among those on the grid.
struct GridSeg {
  int a0, na, b0, key;
};

// Cells that the distances of the atoms [i0, i1) can reach: the cell of
// twice the largest distance from the centre of their box (at most M/2,
// where the period folds).  One CTA, at most 1,024 threads.
__device__ __forceinline__ void grid_extent(const float *__restrict__ pos,
                                            int i0, int i1, float scale,
                                            int half, int *__restrict__ ext) {
  __shared__ float red[32][6];
  __shared__ float mx[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_warps = blockDim.x >> 5;
  float lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) lo[d] = 3e38f, hi[d] = -3e38f;
#pragma unroll 4
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float x = pos[3 * (size_t)i + d];
      lo[d] = fminf(lo[d], x);
      hi[d] = fmaxf(hi[d], x);
    }
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
    if (lane == 0) red[warp][d] = lo[d], red[warp][3 + d] = hi[d];
  }
  __syncthreads();
  float mid[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    float l = red[0][d], h = red[0][3 + d];
    for (int w = 1; w < n_warps; ++w)
      l = fminf(l, red[w][d]), h = fmaxf(h, red[w][3 + d]);
    mid[d] = 0.5f * l + 0.5f * h;
  }
  float r2 = 0.f;
#pragma unroll 4
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    const float x = pos[3 * (size_t)i] - mid[0];
    const float y = pos[3 * (size_t)i + 1] - mid[1];
    const float z = pos[3 * (size_t)i + 2] - mid[2];
    r2 = fmaxf(r2, fmaf(x, x, fmaf(y, y, z * z)));
  }
  for (int o = 16; o > 0; o >>= 1)
    r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, o));
  if (lane == 0) mx[warp] = r2;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < n_warps; ++w) r2 = fmaxf(r2, mx[w]);
    // a millionth more for the roundings here; cells are floor(u).  NaN
    // positions are not seen (their pairs have no cell); with infinite ones
    // every cell is kept
    const float u = 2.000002f * sqrtf(r2) * scale + 2.0f;
    const bool fin = fabsf(mid[0] + mid[1] + mid[2]) < 3e38f;
    *ext = fin && u < (float)half ? (int)u : half;
  }
}

// ext[c] of the configurations on the grid, one CTA each
__global__ void __launch_bounds__(1024)
    grid_extent_kernel(const float *__restrict__ pos,
                       const int *__restrict__ offsets,
                       const int4 *__restrict__ cfg_keys, float scale, int half,
                       int *__restrict__ ext) {
  const int c = cfg_keys[blockIdx.x].x;
  grid_extent(pos, offsets[c], offsets[c + 1], scale, half, ext + blockIdx.x);
}

// How the spreading kernel's warps share the columns, which depends on the
// cells in use and so is known on the device only: CTA b's first `per_cta`
// warps work, warp i = b per_cta + w takes columns [i T / n, (i + 1) T / n).
struct SpreadPlan {
  int used, per_cta, n;
};

constexpr int kSpreadWarps = 16;               // at most, per CTA
constexpr int kSpreadSmem = 224 * 1024;        // of a CTA
constexpr int kSpreadStage = 32 * 32;          // of a warp, beside its cells

struct PlanShape {
  int cell_bytes;  // shared memory per cell and warp
  int min_cols;    // columns that make a warp worth its flush
};

// (all threads of a CTA call this; s: shared scratch of 32 ints)
__device__ __forceinline__ SpreadPlan spread_plan(const int *__restrict__ ext,
                                                  int n_cfgs, int n_ctas,
                                                  PlanShape sh, int total,
                                                  int *s) {
  int u = 0;
  const int t = threadIdx.x;
  for (int i = t; i < n_cfgs; i += blockDim.x) u = max(u, ext[i]);
  u = __reduce_max_sync(0xffffffffu, u);
  if ((t & 31) == 0) s[t >> 5] = u;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  for (int w = 0; w < nw; ++w) u = max(u, s[w]);
  SpreadPlan p;
  p.used = u;
  // as many warps as have room for a histogram
  p.per_cta = min(kSpreadWarps,
                  kSpreadSmem / (kSpreadStage + sh.cell_bytes * grid_words(u)));
  // the four schedulers of the SM get equal numbers of warps
  if (p.per_cta > 4) p.per_cta &= ~3;
  const int per = sh.min_cols * n_ctas;
  p.per_cta = max(1, min(p.per_cta, (total + per - 1) / per));
  p.n = min(p.per_cta * n_ctas, total);  // no warp without a column
  return p;
}

// Where the partial histograms of a launch go.  A warp that leaves a key
// writes its row at slot warp + key (flag 1).  What its last key holds stays
// in shared memory until the CTA is done: if all its warps end on one key,
// their sum is one row of the CTA (cta[b].x = the key, flag 0 at the slots),
// sixteen times less to write and to add up; else each writes its own.
// cta[b].y: whether any warp of CTA b wrote a row of its own.
struct HistRows {
  float *rows;  // [n_ctas] rows of the CTAs, then those of the slots
  int *flag;    // [slots]
  int2 *cta;    // [n_ctas]
  float *low;   // [warps], for sums in float pairs (fq_spread_kernel only)
  int n_ctas, row_words;
  __device__ __forceinline__ float *cta_row(int b) const {
    return rows + (size_t)b * row_words;
  }
  __device__ __forceinline__ float *warp_row(int slot) const {
    return rows + ((size_t)n_ctas + slot) * row_words;
  }
  // what the additions to a warp's row have rounded away so far
  __device__ __forceinline__ float *low_row(int warp) const {
    return low + (size_t)warp * row_words;
  }
};

// x into the float pair (s, c)
__device__ __forceinline__ void pair_add(float x, float &s, float &c) {
  const float y = __fadd_rn(x, c);
  const float t = __fadd_rn(s, y);
  c = __fsub_rn(y, __fsub_rn(t, s));
  s = t;
}

// End of a spreading CTA (all threads call it): whether this warp has to
// write its last key itself.  Else, if s[0] >= 0, the CTA's warps 0 .. s[1]-1
// are to be summed into its row.  s: shared scratch of 32 ints.
__device__ __forceinline__ bool finish_rows(const HistRows &out, int wi,
                                            int key, bool alone, int *s) {
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) s[warp] = key * 2 + alone;
  __syncthreads();
  // (s[w] is negative for warps without work, which come last)
  const int n_warps = blockDim.x >> 5;
  int n = 0, first = s[0] >> 1;
  bool same = true, own = false;
  for (; n < n_warps && s[n] >= 0; ++n) {
    same &= (s[n] >> 1) == first;
    own |= s[n] & 1;
  }
  __syncthreads();
  const bool join = n > 0 && same;
  if (threadIdx.x == 0) {
    out.cta[blockIdx.x] = make_int2(join ? first : -1, own || (n > 0 && !same));
    s[0] = join ? first : -1;
    s[1] = n;
  }
  if (join && key >= 0 && (threadIdx.x & 31) == 0) out.flag[wi + key] = 0;
  __syncthreads();
  return key >= 0 && !join;
}

// One CTA per SM.  Each warp has a private histogram (no atomics, a fixed
// order of additions: the result is the same bits on every run), and the
// columns of all rows, in order, are dealt out evenly to the warps: warp i
// writes one partial histogram per key it meets, at slot i + key.
//
// A column is 32 pairs, one per lane (lane = atom a of the tile, one b):
// distance, cell and weight take about 60 instructions.  They are then
// spread eight pairs at a time: lane = (slot, tap pair), each slot keeping
// its own copy of the histogram, interleaved by cell ([cell][slot]), so that
// the 32 lanes of a read or write fall on 32 different banks whatever the
// cells are, and no two lanes touch the same word.  The lane's two taps of
// the window are polynomials of degree 7 in the pair's position within its
// cell, evaluated together by packed FMAs (coefficients in registers): 19
// instructions per eight pairs.  Bound by instruction issue and the latency
// of its dependent chains (0.59 issued per cycle and scheduler): two columns
// go side by side, and as many warps run as have room for a histogram, 8 per
// SM at 650 cells.  161 instructions per 32 pairs; four slots of one tap per
// lane, at half the memory per warp, took 248.
// 64 x 1,000 atoms at 330 bins: 223 us (fq_pair3_kernel 1,451); 256 alloys of
// 55 to 2,000 atoms at 500 bins 1.22 ms (11.5); 10,007 atoms at 1,500 bins
// 0.47 ms (9.5).
constexpr int kSpreadSlots = 8;
constexpr int kSpreadCols = 2;
constexpr PlanShape kFqPlan{4 * kSpreadSlots, 8};

// the eight copies of word i
__device__ __forceinline__ float sum_copies(const float4 *hist4, int i) {
  const float4 v = hist4[2 * i], w = hist4[2 * i + 1];
  return ((v.x + v.y) + (v.z + v.w)) + ((w.x + w.y) + (w.z + w.w));
}

// Moves a warp's cells to its row, the float pair (row, low) until `last`.
// Not inlined: in line it costs the spreading loop 8 registers and 3 to 6 % of
// its time.
static __device__ __noinline__ void spill_cells(float4 *hist4, float *row,
                                                float *low, int words,
                                                bool add, bool last) {
  __syncwarp();
#pragma unroll 4
  for (int i = threadIdx.x & 31; i < words; i += 32) {
    float s = add ? row[i] : 0.f, c = add ? low[i] : 0.f;
    pair_add(sum_copies(hist4, i), s, c);
    row[i] = last ? s + c : s;
    if (!last) low[i] = c;
    hist4[2 * i] = make_float4(0.f, 0.f, 0.f, 0.f);
    hist4[2 * i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncwarp();
}

// The pairs of a column that the fast distance does not cover (on: the
// lane's is one).  Beyond 128 A they can be most of a call's, so they go
// together as the others do; only those nearer than near_r and those without
// a distance go one at a time.  Not inlined: in line, or as a branch ahead of
// the others' spreading, it costs every call 6 to 24 %.
// 4,000 atoms in two clusters 400 A apart, 500 bins: 426 us (one at a time
// 5,830; fq_pair3_kernel 710).
static __device__ __noinline__ void spread_rest(
    float ahx, float ahy, float ahz, float alx, float aly, float alz,
    float bhx, float bhy, float bhz, float blx, float bly, float blz, bool on,
    float ghi, float glo, float gm, float ginv, float near_r, float near_scale,
    const float *__restrict__ taps, float *hist, int used) {
  if (!__any_sync(0xffffffffu, on)) return;
  const GridScale gs{ghi, glo, gm, ginv};
  const int lane = threadIdx.x & 31, slot = lane >> 2, tp = lane & 3;
  PairDist p{};
  bool wide = on;
  if (on) {
    p = pair_dist_general(ahx + alx, ahy + aly, ahz + alz, bhx + blx,
                          bhy + bly, bhz + blz);
    wide = p.r >= near_r && p.r < 3e38f;
  }
  float uh, ul;
  grid_pos(gs, p.r, p.rl, uh, ul);
  float w = uh < 0.f ? -p.inv_r : p.inv_r;
  ul = uh < 0.f ? -ul : ul;
  uh = fabsf(uh);
  const float fj = floorf(uh);
  // (NaN: the middle of a cell)
  const float t = fminf(fmaxf((uh - fj) + (ul - 0.5f), -0.5f), 0.5f);
  const int j = min(max((int)fj, 0), used);
  if (!wide) w = 0.f;
  for (int src = slot; src < 32; src += 8) {
    float *h = hist + (8 + tp + __shfl_sync(0xffffffffu, j, src)) *
                          kSpreadSlots + slot;
    const float ts = __shfl_sync(0xffffffffu, t, src);
    const float ws = __shfl_sync(0xffffffffu, w, src);
    float f0 = taps[tp * kTapCoef + 7], f1 = taps[(tp + 4) * kTapCoef + 7];
#pragma unroll
    for (int n = 6; n >= 0; --n) {
      f0 = fmaf(f0, ts, taps[tp * kTapCoef + n]);
      f1 = fmaf(f1, ts, taps[(tp + 4) * kTapCoef + n]);
    }
    const float x = h[0], y = h[4 * kSpreadSlots];
    h[0] = x + ws * f0;
    h[4 * kSpreadSlots] = y + ws * f1;
    __syncwarp();
  }
  if (!__any_sync(0xffffffffu, on && !wide)) return;
  for (int l = 0; l < 32; ++l) {
    if (lane == l && on && !wide) {
      if (p.r > 0.f && p.r < near_r) {
        // far below the resolution of Q (Q_max r < 0.6): the power sums of
        // r^2 give sin(Q r)/r, which the window would only give to 1e-7 / r
        const float z = (p.r * near_scale) * (p.r * near_scale);
        float x = 1.f;
        for (int n = 0; n < kNearTerms; ++n, x *= z)
          hist[n * kSpreadSlots] += x;
      } else {
        // r = 0, infinite or NaN: NaN for every bin, as sin(Q r)/r is
        for (int n = 0; n < kTaps; ++n)
          hist[(8 + j + n) * kSpreadSlots] = __int_as_float(0x7fffffff);
      }
    }
    __syncwarp();
  }
}

__global__ void __launch_bounds__(32 * kSpreadWarps)
    fq_spread_kernel(const float *__restrict__ pos,
                     const int *__restrict__ perm,
                     const GridSeg *__restrict__ segs,
                     const int *__restrict__ seg_begin, int n_segs, int total,
                     const int *__restrict__ ext, int n_cfgs, GridScale gs,
                     float near_r, float near_scale,
                     const float *__restrict__ taps, HistRows out) {
  extern __shared__ float4 smem4[];
  __shared__ int splan[32];
  __shared__ bool sspill[kSpreadWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SpreadPlan plan =
      spread_plan(ext, n_cfgs, gridDim.x, kFqPlan, total, splan);
  const int wi = blockIdx.x * plan.per_cta + warp;
  const int c0 = (int)((long long)wi * total / plan.n);
  const int c1 = (int)((long long)(wi + 1) * total / plan.n);
  const bool works = warp < plan.per_cta && wi < plan.n;
  const int words = grid_words(plan.used);
  float4 *stage = smem4 + warp * (kSpreadStage / 16 + 2 * words);
  float4 *hist4 = stage + kSpreadStage / 16;  // [word][slot]
  float *hist = reinterpret_cast<float *>(hist4);
  const int slot = lane >> 2, tp = lane & 3;  // taps tp and tp + 4
  float2 cf[kTapCoef];
#pragma unroll
  for (int i = 0; i < kTapCoef; ++i)
    cf[i] = make_float2(taps[tp * kTapCoef + i], taps[(tp + 4) * kTapCoef + i]);
  for (int i = lane; works && i < 2 * words; i += 32)
    hist4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();
  // the row that holds column c0
  int lo = 0, hi = n_segs;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (seg_begin[mid] <= c0)
      lo = mid;
    else
      hi = mid;
  }
  // tap p of cell j is cell j - 3 + p
  float *const base = hist + (8 + tp) * kSpreadSlots + slot;
  // The cells go to the warp's row when it leaves a key, and after every
  // spill_cols columns: a copy of a cell has then taken about 128 values,
  // where one that grows without limit loses the window's tails.  The row is
  // a float pair, so the sums do not depend on how many columns a warp gets.
  const int spill_cols = 4 * words;
  int since = 0;
  bool spilled = false;
  auto spill = [&](int key, bool last) {
    spill_cells(hist4, out.warp_row(wi + key), out.low_row(wi), words, spilled,
                last);
    if (last && lane == 0) out.flag[wi + key] = 1;
    since = 0;
    spilled = !last;
  };
  int cur = -1;
  bool alone = false;
  int c = c0;
  for (int sgi = lo; works && c < c1; ++sgi) {
    const GridSeg sg = segs[sgi];
    const int begin = seg_begin[sgi], end = min(seg_begin[sgi + 1], c1);
    if (sg.key != cur) {
      if (cur >= 0) {
        spill(cur, true);
        alone = true;
      }
      cur = sg.key;
    }
    // (lanes past the tile count no pair: no b is below 0)
    const int ia = lane < sg.na ? sg.a0 + lane : 0;
    const float4 pa = load_atom(pos, perm, sg.a0 + min(lane, sg.na - 1));
    const SplitAtom a = split_atom(pa.x, pa.y, pa.z);
    for (; c < end; c += 32) {
      // the next 32 (or fewer) b's, staged by one lane each
      const int nb = min(32, end - c);
      const int ib0 = sg.b0 + (c - begin);
      const float4 q = load_atom(pos, perm, ib0 + min(lane, nb - 1));
      const SplitAtom mine = split_atom(q.x, q.y, q.z);
      __syncwarp();
      stage[2 * lane] = make_float4(mine.hx, mine.hy, mine.hz, mine.lx);
      stage[2 * lane + 1] = make_float4(mine.ly, mine.lz, 0.f, 0.f);
      __syncwarp();
      for (int i = 0; i < nb; i += kSpreadCols) {
        // kSpreadCols columns side by side: their chains overlap
        SplitAtom b[kSpreadCols];
        bool on[kSpreadCols], ok[kSpreadCols];
        float t[kSpreadCols], w[kSpreadCols];
        int off[kSpreadCols];
#pragma unroll
        for (int q = 0; q < kSpreadCols; ++q) {
          const int iq = min(i + q, nb - 1);
          const float4 q0 = stage[2 * iq];
          const float2 q1 =
              *reinterpret_cast<const float2 *>(&stage[2 * iq + 1]);
          b[q] = SplitAtom{q0.x, q0.y, q0.z, q0.w, q1.x, q1.y};
          on[q] = ib0 + i + q < ia && i + q < nb;
          PairDist p;
          ok[q] = pair_dist_fast(a, b[q], p) && on[q];
          float uh, ul;
          grid_pos(gs, p.r, p.rl, uh, ul);
          // sin is odd: the half [-M/2, 0] of the period folds on the other
          w[q] = ok[q] ? (uh < 0.f ? -p.inv_r : p.inv_r) : 0.f;
          ul = uh < 0.f ? -ul : ul;
          uh = fabsf(uh);
          const float fj = floorf(uh);
          t[q] = ok[q] ? (uh - fj) + (ul - 0.5f) : 0.f;
          off[q] = ok[q] ? min((int)fj, plan.used) * kSpreadSlots : 0;
        }
        int o[4 * kSpreadCols];
        float2 v[4 * kSpreadCols];
#pragma unroll
        for (int it = 0; it < 4 * kSpreadCols; ++it) {
          const int src = (it & 3) * 8 + slot;
          o[it] = __shfl_sync(0xffffffffu, off[it >> 2], src);
          const float2 tt = f2(__shfl_sync(0xffffffffu, t[it >> 2], src));
          const float2 ww = f2(__shfl_sync(0xffffffffu, w[it >> 2], src));
          float2 f = cf[7];
#pragma unroll
          for (int n = 6; n >= 0; --n) f = __ffma2_rn(f, tt, cf[n]);
          v[it] = __fmul2_rn(ww, f);
        }
#pragma unroll
        for (int it = 0; it < 4 * kSpreadCols; ++it) {
          float *h = base + o[it];
          const float x = h[0], y = h[4 * kSpreadSlots];
          h[0] = x + v[it].x;
          h[4 * kSpreadSlots] = y + v[it].y;
          __syncwarp();
        }
        bool left = false;
#pragma unroll
        for (int q = 0; q < kSpreadCols; ++q) left |= on[q] && !ok[q];
        if (!__any_sync(0xffffffffu, left)) continue;
#pragma unroll
        for (int q = 0; q < kSpreadCols; ++q)
          spread_rest(a.hx, a.hy, a.hz, a.lx, a.ly, a.lz, b[q].hx, b[q].hy,
                      b[q].hz, b[q].lx, b[q].ly, b[q].lz, on[q] && !ok[q],
                      gs.hi, gs.lo, gs.m, gs.inv_m, near_r, near_scale, taps,
                      hist, plan.used);
      }
      since += nb;
      if (since >= spill_cols) spill(cur, false);
    }
    c = end;
  }
  if (lane == 0) sspill[warp] = spilled;
  if (finish_rows(out, wi, works ? cur : -1, alone, splan)) {
    if (spilled) {
      spill(cur, true);
    } else {  // (in line: small batches would wait for the function's code)
      float *row = out.warp_row(wi + cur);
      for (int i = lane; i < words; i += 32) row[i] = sum_copies(hist4, i);
      if (lane == 0) out.flag[wi + cur] = 1;
    }
  } else if (splan[0] >= 0)
    for (int i = threadIdx.x; i < words; i += blockDim.x) {
      float s = 0.f, c = 0.f;
      for (int w = 0; w < splan[1]; ++w) {
        const float x = sum_copies(
            smem4 + w * (kSpreadStage / 16 + 2 * words) + kSpreadStage / 16, i);
        if (sspill[w]) {
          const int wj = blockIdx.x * plan.per_cta + w;
          pair_add(out.warp_row(wj + splan[0])[i], s, c);
          pair_add(out.low_row(wj)[i], s, c);
          pair_add(x, s, c);
        } else {
          s += x;
        }
      }
      out.cta_row(blockIdx.x)[i] = s + c;
    }
}

// The partial histograms of a key: those of columns [c0, c1) at slot offset
// s0, and for ordered species pairs of [d0, d1) at s1.
struct KeyCols {
  int c0, c1, s0, d0, d1, s1;
};

// Sums the partial histograms of a key and folds them for the transform.
// With j' = M/2 - j, sin(2 pi k j'/M) is -(-1)^k sin(2 pi k j/M), so even
// bins need G-_j = H_j - H_j' and odd bins G+_j = H_j + H_j' for j <= M/4
// only: out[j] = (G-_j, G+_j), then the power sums.  The slots follow from
// the plan of the spreading kernel, made again here from its arguments.
// (A key's columns are contiguous, so of the CTAs that hold them only the
// first and the last can hold other keys too.)
// One CTA does cells [nx block, nx (block + 1)); thread (x: cell, y: every
// ny-th row) adds in float pairs, then the thread rows are added in order.
// sred: 4 nx ny floats, splan: 32 ints of shared memory.
__device__ __forceinline__ void fq_grid_reduce(
    const HistRows &in, const KeyCols &kc, const int *__restrict__ ext,
    int n_cfgs, PlanShape shape, int total, int m, int block, int nx, int ny,
    float *__restrict__ out, float *sred, int *splan) {
  const int tid = threadIdx.x;
  const SpreadPlan plan =
      spread_plan(ext, n_cfgs, in.n_ctas, shape, total, splan);
  // the warp of a column
  auto warp_of = [&](long long col) {
    long long i = col * plan.n / total;
    while (i > 0 && i * total / plan.n > col) --i;
    while ((i + 1) * total / plan.n <= col) ++i;
    return (int)i;
  };
  __syncthreads();  // splan has been read
  if (tid < 2) {
    const int c0 = tid ? kc.d0 : kc.c0, c1 = tid ? kc.d1 : kc.c1;
    const int w0 = c0 < c1 ? warp_of(c0) : 0;
    splan[2 * tid] = w0;
    splan[2 * tid + 1] = c0 < c1 ? warp_of(c1 - 1) + 1 : w0;
  }
  __syncthreads();
  const int quarter = m / 4, half = m / 2;
  const int tx = tid % nx, ty = tid / nx;
  const int j = block * nx + tx;
  // the cells that meet in (G-_j, G+_j): j, its mirror images at 0 and M/2
  float hs = 0.f, hc = 0.f, ms = 0.f, mc = 0.f;
  const bool on = j <= quarter, near = j > quarter && j <= quarter + kNearTerms;
  if (ty < ny && (on || near)) {
    const int j1 = half - j, last = plan.used + 4;
    auto take = [&](const float *r) {
      if (near) {
        pair_add(r[j - quarter - 1], hs, hc);
        return;
      }
      r += kGridCell0;
      // cells below 0 and above M/2 are images with the opposite sign
      float x = j <= last ? r[j] : 0.f, y = j1 <= last ? r[j1] : 0.f;
      if (j >= 1 && j <= 3) x -= r[-j];
      if (j >= 1 && half + j <= last) y -= r[half + j];
      pair_add(x, hs, hc);
      pair_add(y, ms, mc);
    };
    auto own = [&](int w, int key) {
      if (in.cta[w / plan.per_cta].y && in.flag[w + key])
        take(in.warp_row(w + key));
    };
    for (int part = 0; part < 2; ++part) {
      const int w0 = splan[2 * part], w1 = splan[2 * part + 1];
      if (w0 == w1) continue;
      const int key = part ? kc.s1 : kc.s0;
      const int b0 = w0 / plan.per_cta, b1 = (w1 - 1) / plan.per_cta;
#pragma unroll 2
      for (int b = b0 + ty; b <= b1; b += ny)
        if (in.cta[b].x == key) take(in.cta_row(b));
      // warps that wrote their own row
      {
        const int e0 = min(w1, (b0 + 1) * plan.per_cta);
        for (int w = w0 + ty; w < e0; w += ny) own(w, key);
        for (int w = max(e0, b1 * plan.per_cta) + ty; w < w1; w += ny)
          own(w, key);
      }
    }
  }
  const int st = nx * ny;
  if (ty < ny) {
    float *sh = sred + tid;
    sh[0] = hs;
    sh[st] = hc;
    sh[2 * st] = ms;
    sh[3 * st] = mc;
  }
  __syncthreads();
  if (ty != 0 || !(on || near)) return;
  for (int y = 1; y < ny; ++y) {
    const float *sh = sred + y * nx + tx;
    pair_add(sh[0], hs, hc);
    hc += sh[st];
    pair_add(sh[2 * st], ms, mc);
    mc += sh[3 * st];
  }
  if (near) {
    out[2 * (quarter + 1) + (j - quarter - 1)] = hs + hc;
  } else {
    const bool mid = j == quarter;  // its own mirror image
    out[2 * j] = j == 0 || mid ? 0.f : (hs - ms) + (hc - mc);
    out[2 * j + 1] = j == 0 ? 0.f : mid ? hs + hc : (hs + ms) + (hc + mc);
  }
}

// floats of one key's sums (even, so that the pairs stay 8-byte aligned)
__host__ __device__ constexpr int fq_sum_floats(int m) {
  return 2 * (m / 4 + 1) + 8;
}
__host__ __device__ constexpr int fq_reduce_blocks(int m, int nx) {
  return (m / 4 + kNearTerms) / nx + 1;
}

__global__ void fq_grid_reduce_kernel(HistRows in,
                                      const KeyCols *__restrict__ key_cols,
                                      const int *__restrict__ ext, int n_cfgs,
                                      PlanShape shape, int total, int m, int nx,
                                      int ny, float *__restrict__ out) {
  extern __shared__ float sred[];
  __shared__ int splan[32];
  fq_grid_reduce(in, key_cols[blockIdx.y], ext, n_cfgs, shape, total, m,
                 blockIdx.x, nx, ny,
                 out + (size_t)blockIdx.y * fq_sum_floats(m), sred, splan);
}

// Sum over a key's near pairs of sin(Q r)/r = Q sum_n (-1)^n (Q r)^2n /
// (2n + 1)!; nr[n] = sum (Q_max r)^2n, near_unit = 1 / n_bins.
__device__ __forceinline__ double near_sum(const float *nr, int k,
                                           float near_unit, double dq) {
  if (nr[0] == 0.f) return 0.0;
  const float z = -(k * near_unit) * (k * near_unit);
  const float v =
      nr[0] + z * (nr[1] / 6.f +
                   z * (nr[2] / 120.f +
                        z * (nr[3] / 5040.f + z * (nr[4] / 362880.f))));
  return (double)k * dq * (double)v;
}

// F(Q) of the configurations on the grid.  CTA = (32 bins, configuration),
// lane = bin k.  sum_j G_j sin(theta_k j) goes in blocks of 2 R + 1 cells
// around a centre c: sin(theta (c +- n)) = sin(theta c) cos(theta n) +-
// cos(theta c) sin(theta n), so a block is
//   sin(theta c) sum_n cos(theta n) (G_c+n + G_c-n)
//   + cos(theta c) sum_n sin(theta n) (G_c+n - G_c-n)
// with the sums and differences formed once per CTA as the cells are staged
// in shared memory, and the rotations of n <= R kept in registers: 1.5
// instructions per (bin, cell) and one accurate sine and cosine per block.
// The warps share the blocks; block sums are added in float pairs, the rest
// is FP64 per bin.  Four keys at a time, so that their copies and barriers
// are waited for once.
constexpr int kFqDftWarps = 8;
constexpr int kFqDftReach = 16;
constexpr int kFqDftKeys = 4;
__host__ __device__ constexpr int fq_dft_blocks(int m) {
  return (m / 4 + 2 * kFqDftReach) / (2 * kFqDftReach + 1);
}
// float4 of shared memory, per key: (sum, difference) of even bins, then of
// odd ones
__host__ __device__ constexpr int fq_dft_float4(int m) {
  return kFqDftKeys * fq_dft_blocks(m) * (kFqDftReach + 1);
}
__global__ void __launch_bounds__(32 * kFqDftWarps, 3)
    fq_grid_finish_kernel(const float *__restrict__ hsum,
                          const int4 *__restrict__ cfg_keys,
                          const int *__restrict__ key_spair,
                          const int2 *__restrict__ spair_species,
                          const float *__restrict__ ftab,
                          const double *__restrict__ na,
                          const double *__restrict__ inv_phi, int m,
                          float inv_m, int n_bins, int kb_out, double dq,
                          float near_unit, float *__restrict__ fq,
                          double *__restrict__ fq_raw) {
  constexpr int R = kFqDftReach, B = 2 * R + 1, Q = kFqDftKeys;
  extern __shared__ float4 sh4[];
  __shared__ float red[Q][2][kFqDftWarps][32];
  __shared__ double terms[Q][32];
  const int4 ck = cfg_keys[blockIdx.y];  // configuration, first key, keys
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = min((int)(blockIdx.x * 32 + lane), n_bins - 1);
  const int quarter = m / 4, blocks = fq_dft_blocks(m);
  // e^{i theta n}: each fourth from the table's accuracy, the rest one
  // product each
  float sn[R + 1], cn[R + 1];
  sn[0] = 0.f;
  cn[0] = 1.f;
#pragma unroll
  for (int n = 1; n <= R; ++n) {
    const int r = n & 3;
    if (r == 0 || n < 4) {
      sincos_turn((int)((unsigned)n * (unsigned)k % (unsigned)m), m, inv_m,
                  sn[n], cn[n]);
    } else {
      sn[n] = fmaf(sn[n - r], cn[r], cn[n - r] * sn[r]);
      cn[n] = fmaf(cn[n - r], cn[r], -sn[n - r] * sn[r]);
    }
  }
  double sum = 0.0;
  for (int q0 = 0; q0 < ck.z; q0 += Q) {
    const int nq = min(Q, ck.z - q0), per = blocks * (R + 1);
    const float *hq = hsum + (size_t)(ck.y + q0) * fq_sum_floats(m);
    __syncthreads();
    for (int i = threadIdx.x; i < nq * per; i += blockDim.x) {
      const int q = i / per, b = (i - q * per) / (R + 1);
      const int n = i - q * per - b * (R + 1);
      const float *h = hq + (size_t)q * fq_sum_floats(m);
      const int jp = 1 + b * B + R + n, jm = 1 + b * B + R - n;
      float2 p = make_float2(0.f, 0.f), o = p;
      if (jp <= quarter) p = *reinterpret_cast<const float2 *>(h + 2 * jp);
      if (n > 0 && jm <= quarter)
        o = *reinterpret_cast<const float2 *>(h + 2 * jm);
      sh4[i] = make_float4(p.x + o.x, p.x - o.x, p.y + o.y, p.y - o.y);
    }
    __syncthreads();
    for (int q = 0; q < nq; ++q) {
      const float2 *hk =
          reinterpret_cast<const float2 *>(sh4 + q * per) + (k & 1);
      float s = 0.f, c = 0.f;
      // (the warps take turns at who gets one block more)
      for (int b = (warp + q * blocks) % kFqDftWarps; b < blocks;
           b += kFqDftWarps) {
        float sc, cc;
        sincos_turn(
            (int)((unsigned)k * (unsigned)(1 + b * B + R) % (unsigned)m), m,
            inv_m, sc, cc);
        float u = 0.f, v = 0.f;
#pragma unroll
        for (int n = 0; n <= R; ++n) {
          const float2 x = hk[2 * (b * (R + 1) + n)];
          u = fmaf(cn[n], x.x, u);
          v = fmaf(sn[n], x.y, v);
        }
        pair_add(fmaf(sc, u, cc * v), s, c);
      }
      red[q][0][warp][lane] = s;
      red[q][1][warp][lane] = c;
    }
    __syncthreads();
    if (warp < nq) {  // one key per warp
      float s = 0.f, c = 0.f;
      for (int w = 0; w < kFqDftWarps; ++w) {
        const float y = __fadd_rn(red[warp][0][w][lane], c);
        const float t = __fadd_rn(s, y);
        c = __fsub_rn(y, __fsub_rn(t, s)) + red[warp][1][w][lane];
        s = t;
      }
      const double d =
          ((double)s + (double)c) * inv_phi[k] +
          near_sum(hq + (size_t)warp * fq_sum_floats(m) + 2 * (quarter + 1), k,
                   near_unit, dq);
      const int2 ss = spair_species[key_spair[ck.y + q0 + warp]];
      terms[warp][lane] = (double)ftab[ss.x * n_bins + k] *
                          (double)ftab[ss.y * n_bins + k] * d;
    }
    __syncthreads();
    if (warp == 0)
      for (int q = 0; q < nq; ++q) sum += terms[q][lane];
  }
  const int kk = blockIdx.x * 32 + lane;
  if (warp != 0 || kk >= n_bins) return;
  const size_t o = (size_t)ck.x * n_bins + kk;
  const bool on = kk >= kb_out;
  if (fq) fq[o] = on ? fq_value(sum, na[o]) : 0.f;
  if (fq_raw) fq_raw[o] = on ? sum : 0.0;
}

// The same transform in FP64 for configurations of many pairs.  The rotations
// by n cells are common to all blocks of a bin, so what FP32 rounds off them
// multiplies every 33rd cell's sum, which sees the small-angle peak of F (its
// height grows with the atoms) at the bins near multiples of M / 33.
// Above 1e8 pairs, where the direct kernels' error is passed (error of F at
// 20,000 atoms 2.0e-7 in FP32, 6.3e-8 so, direct 1.5e-7; at 14,000 1.2e-7 in
// FP32, direct 1.8e-7).
// One key at a time; warps share the blocks, each centre one rotation by
// kFqDftWarps blocks from the one before.  FP64 bound: 38 us at 1,500 bins,
// of 1.4 ms and more.
__host__ __device__ constexpr int fq_wide_smem(int m) {
  return fq_dft_blocks(m) * (kFqDftReach + 1) * 4 * (int)sizeof(double);
}
__global__ void __launch_bounds__(32 * kFqDftWarps)
    fq_grid_finish_wide_kernel(const float *__restrict__ hsum,
                               const int4 *__restrict__ cfg_keys,
                               const int *__restrict__ key_spair,
                               const int2 *__restrict__ spair_species,
                               const float *__restrict__ ftab,
                               const double *__restrict__ na,
                               const double *__restrict__ inv_phi, int m,
                               int n_bins, int kb_out, double dq,
                               float near_unit, float *__restrict__ fq,
                               double *__restrict__ fq_raw) {
  constexpr int R = kFqDftReach, B = 2 * R + 1;
  extern __shared__ double2 sh2[];  // [block][n][even, odd bins]
  __shared__ double red[kFqDftWarps][32];
  const int4 ck = cfg_keys[blockIdx.y];  // configuration, first key, keys
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = min((int)(blockIdx.x * 32 + lane), n_bins - 1);
  const int quarter = m / 4, blocks = fq_dft_blocks(m);
  auto turn = [&](int n, double &s, double &c) {  // of 2 pi k n / m
    sincospi(2.0 * (double)((unsigned)n * (unsigned)k % (unsigned)m) /
                 (double)m,
             &s, &c);
  };
  double s1, c1, sw, cw, s0, c0;
  turn(1, s1, c1);
  turn(B * kFqDftWarps % m, sw, cw);
  turn((1 + warp * B + R) % m, s0, c0);
  double sum = 0.0;
  for (int q = 0; q < ck.z; ++q) {
    const float *h = hsum + (size_t)(ck.y + q) * fq_sum_floats(m);
    __syncthreads();
    for (int i = threadIdx.x; i < blocks * (R + 1); i += blockDim.x) {
      const int b = i / (R + 1), n = i - b * (R + 1);
      const int jp = 1 + b * B + R + n, jm = 1 + b * B + R - n;
      float2 p = make_float2(0.f, 0.f), o = p;
      if (jp <= quarter) p = *reinterpret_cast<const float2 *>(h + 2 * jp);
      if (n > 0 && jm <= quarter)
        o = *reinterpret_cast<const float2 *>(h + 2 * jm);
      sh2[2 * i] = make_double2((double)p.x + o.x, (double)p.x - o.x);
      sh2[2 * i + 1] = make_double2((double)p.y + o.y, (double)p.y - o.y);
    }
    __syncthreads();
    const double2 *hk = sh2 + (k & 1);
    double s = 0.0, sc = s0, cc = c0;
    for (int b = warp; b < blocks; b += kFqDftWarps) {
      double u = 0.0, v = 0.0, sn = 0.0, cn = 1.0;
#pragma unroll
      for (int n = 0; n <= R; ++n) {
        const double2 x = hk[2 * (b * (R + 1) + n)];
        u = fma(cn, x.x, u);
        v = fma(sn, x.y, v);
        const double t = fma(sn, c1, cn * s1);
        cn = fma(cn, c1, -sn * s1);
        sn = t;
      }
      s += fma(sc, u, cc * v);
      const double t = fma(sc, cw, cc * sw);
      cc = fma(cc, cw, -sc * sw);
      sc = t;
    }
    red[warp][lane] = s;
    __syncthreads();
    if (warp == 0) {
      s = 0.0;
      for (int w = 0; w < kFqDftWarps; ++w) s += red[w][lane];
      const int2 ss = spair_species[key_spair[ck.y + q]];
      sum += (double)ftab[ss.x * n_bins + k] *
             (double)ftab[ss.y * n_bins + k] *
             (s * inv_phi[k] +
              near_sum(h + 2 * (quarter + 1), k, near_unit, dq));
    }
  }
  const int kk = blockIdx.x * 32 + lane;
  if (warp != 0 || kk >= n_bins) return;
  const size_t o = (size_t)ck.x * n_bins + kk;
  const bool on = kk >= kb_out;
  if (fq) fq[o] = on ? fq_value(sum, na[o]) : 0.f;
  if (fq_raw) fq_raw[o] = on ? sum : 0.0;
}

}  // namespace pyiid
