// grad_grid.cuh -- dF/dx (and F(Q) beside it) by spreading each atom's pairs
// on a phase grid and transforming the grid to the bins.
//
// Row a of the reference-convention gradient (cpu_flat.py:122-194 with the
// scatter signs of cpu_experimental.py:8-15, pyiid/experiments/
// elasticscatter/kernels) is, per species of b,
//   -(f_a f_b / na) sum_b (x_a - x_b) (Q cos(Q r) - sin(Q r)/r) / r^2.
// With w = (x_a - x_b)/r^3 and S(theta) = sum_b w sin(theta u), theta = 2 pi
// k / M and u = r M dq / (2 pi), the sum over b is theta S'(theta) - S(theta).
// As in fq_grid.cuh the pairs go on the grid with a window,
//   H_j = sum_b w phi(j - u),  sum_j H_j sin(theta j) = phihat(theta) S,
// and the derivative of that identity gives S' from the same H:
//   g = P_k X_k - R_k Y_k,   X = sum_j j H_j cos(theta j),
//   Y = sum_j H_j sin(theta j),  P = theta / phihat,
//   R = (1 + theta phihat' / phihat) / phihat.
// So a row costs one real transform of length M per coordinate and species
// instead of N n_bins terms, and a pair one histogram update.
#pragma once

#include "debye_kernels.cuh"
#include "fq_grid.cuh"
#include "phase_grid.cuh"

namespace pyiid {

// Units of one (species of a, species of b) in one part of the atoms: unit u is
// atom a0 + u against the n_b atoms from b0, in cols columns of 32.  Columns
// of a part's units are numbered block after block from col0.
// s_a, s_b: where the species' atoms start in the array of grad_prep_kernel;
// atom a0 is number i_a of the cols_a x 32 there.
struct GradBlock {
  int col0, cols, unit0, a0, n_a, b0, n_b, s_a, s_b, i_a, cols_a;
};

__device__ __forceinline__ SplitAtom staged_atom(const float4 &p,
                                                 const float4 &q) {
  return SplitAtom{p.x, p.y, p.z, p.w, q.x, q.y};
}

// One launch for what the gradient needs beforehand.  The first CTA finds
// the cells in use (as grid_extent_kernel), the others write the
// coefficients coef[sa][sb][k] = -f_sa f_sb / na_k and the split atoms of
// each species in the order of its columns: lane l of column c is atom
// c + l cols.  Neighbours in the caller's list are often neighbours in a
// shell and would fall on the same cells; a column takes every cols-th
// atom (four pairs collide in 9 % of the groups instead of 19 at 20,000
// atoms of a particle listed by shells, in 31 % instead of 36 at 1,000).
constexpr int kPrepBlock = 512;
__global__ void __launch_bounds__(kPrepBlock)
    grad_prep_kernel(const float *__restrict__ pos, const int *__restrict__ perm,
                     int n, const GradBlock *__restrict__ blocks,
                     int n_species, float scale, int half,
                     int *__restrict__ ext, const double *__restrict__ na,
                     const float *__restrict__ ftab, int n_bins,
                     float *__restrict__ coef, float4 *__restrict__ atoms) {
  if (blockIdx.x == 0) {
    grid_extent(pos, 0, n, scale, half, ext);
    return;
  }
  const int first = (blockIdx.x - 1) * kPrepBlock + threadIdx.x;
  const int stride = (gridDim.x - 1) * kPrepBlock;
  for (int i = first; i < n_species * n_species * n_bins; i += stride) {
    const int k = i % n_bins, s = i / n_bins;
    const int sa = s / n_species, sb = s % n_species;
    const float nak = (float)na[k];
    coef[i] = -(ftab[sa * n_bins + k] * ftab[sb * n_bins + k]) / nak;
  }
  for (int sp = 0; sp < n_species; ++sp) {
    const GradBlock B = blocks[sp];  // species 0 against sp
    const int cols = (B.n_b + 31) / 32;
    for (int i = first; i < cols * 32; i += stride) {
      const int b = min((i >> 5) + (i & 31) * cols, B.n_b - 1);
      const float4 p = load_atom(pos, perm, B.b0 + b);
      const SplitAtom a = split_atom(p.x, p.y, p.z);
      atoms[2 * (B.s_b + i)] = make_float4(a.hx, a.hy, a.hz, a.lx);
      atoms[2 * (B.s_b + i) + 1] = make_float4(a.ly, a.lz, 0.f, 0.f);
    }
  }
}

// (x, y, z, F) of one cell; a warp's flush costs about two columns
constexpr PlanShape kGradPlan{16, 4};

// A word of shared memory by its 32-bit address; volatile, so that the order
// of a warp's updates is the program's.
__device__ __forceinline__ float lds(int addr) {
  float x;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(addr) : "memory");
  return x;
}
__device__ __forceinline__ void sts(int addr, float x) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(x) : "memory");
}

// A staged column: weights [4][32 + 4] (x, y, z, F; the four rows on different
// banks), shared-memory words of the cells [32], positions [32].
__device__ __forceinline__ void stage_column(float *sw, int hbase, int cell,
                                             float t, float x, float y, float z,
                                             float f) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  sw[lane] = x;
  sw[36 + lane] = y;
  sw[72 + lane] = z;
  sw[108 + lane] = f;
  reinterpret_cast<int *>(sw)[144 + lane] = hbase + cell * 16;
  sw[176 + lane] = t;
  __syncwarp();
}

// Bit of each lane whose group of four has cells that overlap.
__device__ __forceinline__ unsigned tied_groups(int cell) {
  bool near4 = false;
#pragma unroll
  for (int x = 1; x < 4; ++x)
    near4 |= abs(__shfl_xor_sync(0xffffffffu, cell, x) - cell) < kTaps;
  return __ballot_sync(0xffffffffu, near4);
}

// Adds a staged column to the warp's cells, lane = (tap, component).
__device__ __forceinline__ void spread_column(const float *sw, unsigned tied,
                                              const float2 (&cf)[kTapCoef]) {
  const int lane = threadIdx.x & 31;
  const int4 *so4 = reinterpret_cast<const int4 *>(sw + 144);
  const float4 *st4 = reinterpret_cast<const float4 *>(sw + 176);
  const float4 *sw4 = reinterpret_cast<const float4 *>(sw) + 9 * (lane & 3);
  int4 no = so4[0];
  float4 nt = st4[0], nv = sw4[0];
#pragma unroll 2
  for (int g = 0; g < 8; ++g) {
    const int4 o = no;
    const float4 t4 = nt, v = nv;
    // (the last one reads what lies behind, inside the warp's stage)
    no = so4[g + 1];
    nt = st4[g + 1];
    nv = sw4[g + 1];
    const float2 t01 = make_float2(t4.x, t4.y);
    const float2 t23 = make_float2(t4.z, t4.w);
    float2 f01 = cf[7], f23 = cf[7];
#pragma unroll
    for (int m = 6; m >= 0; --m) {
      f01 = __ffma2_rn(f01, t01, cf[m]);
      f23 = __ffma2_rn(f23, t23, cf[m]);
    }
    const int h0 = o.x + 4 * lane, h1 = o.y + 4 * lane;
    const int h2 = o.z + 4 * lane, h3 = o.w + 4 * lane;
    if ((tied >> (4 * g)) & 0xfu) {
      sts(h0, fmaf(v.x, f01.x, lds(h0)));
      __syncwarp();
      sts(h1, fmaf(v.y, f01.y, lds(h1)));
      __syncwarp();
      sts(h2, fmaf(v.z, f23.x, lds(h2)));
      __syncwarp();
      sts(h3, fmaf(v.w, f23.y, lds(h3)));
    } else {
      const float x0 = lds(h0), x1 = lds(h1), x2 = lds(h2), x3 = lds(h3);
      sts(h0, fmaf(v.x, f01.x, x0));
      sts(h1, fmaf(v.y, f01.y, x1));
      sts(h2, fmaf(v.z, f23.x, x2));
      sts(h3, fmaf(v.w, f23.y, x3));
    }
    __syncwarp();
  }
}

// The pairs of a column that the fast distance does not cover, as spread_rest
// of fq_grid.cuh; returns whether the lane's pair is a period or more away.
// The two clusters named there, F and dF/dx: 1,807 us (one at a time 8,076,
// fqgrad2_kernel 3,352).
// stage: the warp's, as grad_spread_kernel lays it out.
template <bool WITH_F>
static __device__ __noinline__ bool grad_spread_rest(
    float ahx, float ahy, float ahz, float alx, float aly, float alz,
    float bhx, float bhy, float bhz, float blx, float bly, float blz, bool on,
    int sweep, float ghi, float glo, float gm, float ginv, float near_r,
    float near_scale, const float *__restrict__ taps, float4 *stage,
    float4 *hist4, int used) {
  const GridScale gs{ghi, glo, gm, ginv};
  const int lane = threadIdx.x & 31;
  PairDist p{};
  bool use = on;
  if (on) {
    p = pair_dist_general(ahx + alx, ahy + aly, ahz + alz, bhx + blx,
                          bhy + bly, bhz + blz);
    use = p.r >= near_r && p.r < 3e38f;
  }
  float uh, ul;
  const float n = grid_pos(gs, p.r, p.rl, uh, ul);
  const float s = uh < 0.f ? -1.0f : 1.0f;
  const float ua = fabsf(uh), fj = floorf(ua);
  // (NaN: the middle of a cell)
  const float t = fminf(fmaxf((ua - fj) + (s * ul - 0.5f), -0.5f), 0.5f);
  const int j = min(max((int)fj, 0), used);
  const float w =
      (p.inv_r * p.inv_r) * (sweep ? gs.m * n * p.inv_r : s * p.inv_r);
  float2 cf[kTapCoef];
#pragma unroll
  for (int i = 0; i < kTapCoef; ++i)
    cf[i] = f2(taps[(lane >> 2) * kTapCoef + i]);
  float *const sw = reinterpret_cast<float *>(stage);
  stage_column(sw, (int)__cvta_generic_to_shared(hist4 + 8), j, t,
               use ? w * p.dx : 0.f, use ? w * p.dy : 0.f,
               use ? w * p.dz : 0.f,
               use && WITH_F && !sweep ? 0.5f * s * p.inv_r : 0.f);
  spread_column(sw, tied_groups(j), cf);
  for (unsigned rest = __ballot_sync(0xffffffffu, on && !use); rest;
       rest &= rest - 1) {
    if (lane == __ffs(rest) - 1) {
      if (p.r > 0.f && p.r < near_r) {
        // far below the resolution of Q: power sums of r^2
        const float z = (p.r * near_scale) * (p.r * near_scale);
        float x = sweep ? 0.f : 1.f;
        for (int m = 0; m < kNearTerms; ++m, x *= z) {
          hist4[m].x += x * p.dx;
          hist4[m].y += x * p.dy;
          hist4[m].z += x * p.dz;
          if (WITH_F) hist4[m].w += 0.5f * x;
        }
      } else {
        // r = 0, infinite or NaN: NaN for every bin
        const float bad = __int_as_float(0x7fffffff);
        for (int m = 0; m < kTaps; ++m) {
          float4 &x = hist4[8 + j + m];
          x.x = x.y = x.z = bad;
          if (WITH_F) x.w = bad;
        }
      }
    }
    __syncwarp();
  }
  return use && n != 0.f;
}

// One CTA per SM, each warp with a private histogram; the columns of all
// units, in order, are dealt out evenly to the warps (spread_plan), so a unit
// may be cut between warps: warp i writes its part of unit u at row i + u,
// and the transform adds the parts (parts[u]: the first and the last warp of
// unit u).  No atomics: the same bits on every run.
//
// A column is one atom a against 32 b's, one per lane: distance, cell,
// weights.  The pairs are then spread one at a time, lane = (tap, component):
// the 8 cells x (x, y, z, F) of a pair are 32 consecutive words.  What a warp
// waits for is the chain read - add - write, so four pairs go together when
// no two of them are within 8 cells (found for all groups of four by three
// shuffles), one by one otherwise.  Bound by the shared-memory pipe (82 %
// busy; 16.2 instructions per ordered pair fill 64 % of the issue slots, both
// counted at the 2,001 atoms below).
// 2,001 atoms, 4.0 M ordered pairs, without F: 90 us; 20,000 atoms with F,
// 400 M pairs: 9.8 ms (gradfq2_kernel 2,056 us, fqgrad2_kernel 205 ms, whose
// work grows with the bins too).
// With WITH_F the fourth word collects sin(Q r)/r (half of each ordered
// pair) over all units of a block; finish_rows joins a CTA's partial sums.
//
// X needs the true distance of a pair, not the one folded into half a
// period, r = s r_folded + n P: the rows hold s w, and where any n is not 0
// a second sweep writes the rows of n M w to rows2 (flag[row] = 1), which
// the transform adds to j H_j.
template <bool WITH_F>
__global__ void __launch_bounds__(32 * kSpreadWarps)
    grad_spread_kernel(const float4 *__restrict__ atoms,
                       const GradBlock *__restrict__ blocks, int total,
                       const int *__restrict__ ext, GridScale gs, float near_r,
                       float near_scale, const float *__restrict__ taps,
                       float *__restrict__ rows, float *__restrict__ rows2,
                       int *__restrict__ flag, int2 *__restrict__ parts,
                       HistRows fout) {
  extern __shared__ float4 smem4[];
  __shared__ int splan[32];
  __shared__ bool sspill[kSpreadWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SpreadPlan plan =
      spread_plan(ext, 1, gridDim.x, kGradPlan, total, splan);
  const int wi = blockIdx.x * plan.per_cta + warp;
  const int c0 = (int)((long long)wi * total / plan.n);
  const int c1 = (int)((long long)(wi + 1) * total / plan.n);
  const bool works = warp < plan.per_cta && wi < plan.n;
  const int words = grid_words(plan.used);
  float4 *const stage = smem4 + warp * (kSpreadStage / 16 + words);
  float *const sw = reinterpret_cast<float *>(stage);
  float4 *const hist4 = stage + kSpreadStage / 16;  // [word]
  const int hbase = (int)__cvta_generic_to_shared(hist4 + 8);
  float2 cf[kTapCoef];
#pragma unroll
  for (int i = 0; i < kTapCoef; ++i) cf[i] = f2(taps[(lane >> 2) * kTapCoef + i]);
  for (int i = lane; works && i < words; i += 32)
    hist4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();
  // F goes to the warp's row at the end of a block, and every kSpillCols
  // columns before: a cell that has grown to hundreds of pairs would lose the
  // window's tails (6e-7 of F at 20,000 atoms without, 2e-7 so)
  constexpr int kSpillCols = 1024;
  int since = 0;
  bool spilled = false;
  auto spill_f = [&](int key) {
    __syncwarp();
    float *out = fout.warp_row(wi + key);
    for (int i = lane; i < words; i += 32) {
      out[i] = spilled ? out[i] + hist4[i].w : hist4[i].w;
      hist4[i].w = 0.f;
    }
    since = 0;
    spilled = true;
    __syncwarp();
  };
  auto flush_f = [&](int key) {
    spill_f(key);
    spilled = false;
    if (lane == 0) fout.flag[wi + key] = 1;
  };
  int bi = 0;
  bool alone = false;
  if (works)
    while (c0 >= blocks[bi].col0 + blocks[bi].cols * blocks[bi].n_a) ++bi;
  GradBlock B = blocks[bi];
  for (int c = c0; works && c < c1;) {
    if (c >= B.col0 + B.cols * B.n_a) {
      if (WITH_F) {
        flush_f(bi);
        alone = true;
      }
      do {
        B = blocks[++bi];
      } while (c >= B.col0 + B.cols * B.n_a);
    }
    const int u = (c - B.col0) / B.cols;
    const int cb = c - B.col0 - u * B.cols;
    const int ce = min(B.cols, cb + (c1 - c));
    const int ia = B.a0 + u;
    // atom a in the order of the columns (see grad_prep_kernel)
    const int ua = B.i_a + u;
    const float4 *pa =
        atoms + 2 * (B.s_a + (ua % B.cols_a) * 32 + ua / B.cols_a);
    const SplitAtom a = staged_atom(pa[0], pa[1]);
    const size_t row = (size_t)(wi + B.unit0 + u) * 3 * words;
    bool wide = false;
    for (int sweep = 0; sweep < 2; ++sweep) {
      const float4 *pb = atoms + 2 * (B.s_b + cb * 32 + lane);
      float4 q0 = pb[0], q1 = pb[1];
      for (int col = cb; col < ce; ++col) {
        const SplitAtom b = staged_atom(q0, q1);
        const int jb = col + lane * B.cols;
        pb += 64;
        if (col + 1 < ce) {
          q0 = pb[0];
          q1 = pb[1];
        }
        const bool on = jb < B.n_b && B.b0 + jb != ia;
        PairDist p;
        const bool ok = pair_dist_fast(a, b, p) && on;
        float uh, ul;
        const float n = grid_pos(gs, p.r, p.rl, uh, ul);
        wide |= ok && n != 0.f;
        const float sg = uh < 0.f ? -1.0f : 1.0f;
        float w = (p.inv_r * p.inv_r) * (sweep ? gs.m * n * p.inv_r
                                               : sg * p.inv_r);
        float wf = WITH_F && !sweep ? 0.5f * sg * p.inv_r : 0.f;
        const float ua = fabsf(uh), fj = floorf(ua);
        const float t = ok ? (ua - fj) + (sg * ul - 0.5f) : 0.f;
        const int cell = ok ? min((int)fj, plan.used) : 0;
        stage_column(sw, hbase, cell, t, ok ? w * p.dx : 0.f,
                     ok ? w * p.dy : 0.f, ok ? w * p.dz : 0.f, ok ? wf : 0.f);
        spread_column(sw, tied_groups(cell), cf);
        if (!__any_sync(0xffffffffu, on && !ok)) continue;
        wide |= grad_spread_rest<WITH_F>(
            a.hx, a.hy, a.hz, a.lx, a.ly, a.lz, b.hx, b.hy, b.hz, b.lx, b.ly,
            b.lz, on && !ok, sweep, gs.hi, gs.lo, gs.m, gs.inv_m, near_r,
            near_scale, taps, stage, hist4, plan.used);
      }
      __syncwarp();
      float *out = (sweep ? rows2 : rows) + row;
      for (int i = lane; i < words; i += 32) {
        const float4 v = hist4[i];
        out[i] = v.x;
        out[words + i] = v.y;
        out[2 * words + i] = v.z;
        hist4[i] = make_float4(0.f, 0.f, 0.f, v.w);
      }
      __syncwarp();
      if (sweep) break;
      wide = __any_sync(0xffffffffu, wide);
      if (lane == 0) {
        flag[wi + B.unit0 + u] = wide;
        if (cb == 0) parts[B.unit0 + u].x = wi;
        if (ce == B.cols) parts[B.unit0 + u].y = wi;
      }
      if (!wide) break;
    }
    c += ce - cb;
    since += ce - cb;
    if (WITH_F && since >= kSpillCols) spill_f(bi);
  }
  if (WITH_F) {
    if (lane == 0) sspill[warp] = spilled;
    if (finish_rows(fout, wi, works ? bi : -1, alone, splan))
      flush_f(bi);
    else if (splan[0] >= 0)
      for (int i = threadIdx.x; i < words; i += blockDim.x) {
        float s = 0.f;
        for (int w = 0; w < splan[1]; ++w) {
          s += smem4[(w + 1) * (kSpreadStage / 16) + w * words + i].w;
          if (sspill[w])
            s += fout.warp_row(blockIdx.x * plan.per_cta + w + splan[0])[i];
        }
        fout.cta_row(blockIdx.x)[i] = s;
      }
  }
}

// ------------------------------------------------------------- transform
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  return make_float2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return make_float2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 mul_mi(float2 a) {  // -i a
  return make_float2(a.y, -a.x);
}

// In-place discrete Fourier transforms (e^{-2 pi i / R}) of R values, built
// from the ones of two, three and four by the Cooley-Tukey split R = P Q:
// v[Q p + q] in, bin p' + P q' out at v[P q' + p'].
__device__ __forceinline__ void dft2(float2 &a, float2 &b) {
  const float2 t = csub(a, b);
  a = cadd(a, b);
  b = t;
}
__device__ __forceinline__ void dft3(float2 &a, float2 &b, float2 &c) {
  constexpr float kS = 0.86602540378f;  // sin(2 pi / 3)
  const float2 s = cadd(b, c), d = csub(b, c);
  const float2 m = make_float2(fmaf(-0.5f, s.x, a.x), fmaf(-0.5f, s.y, a.y));
  a = cadd(a, s);
  b = make_float2(fmaf(kS, d.y, m.x), fmaf(-kS, d.x, m.y));
  c = make_float2(fmaf(-kS, d.y, m.x), fmaf(kS, d.x, m.y));
}
__device__ __forceinline__ void dft4(float2 &a, float2 &b, float2 &c,
                                     float2 &d) {
  dft2(a, c);
  dft2(b, d);
  d = mul_mi(d);
  dft2(a, b);  // bins 0, 2
  dft2(c, d);  // bins 1, 3
  const float2 t = b;
  b = c;
  c = t;
}

template <int R>
__device__ __forceinline__ void dft(float2 (&v)[R]);

template <>
__device__ __forceinline__ void dft<4>(float2 (&v)[4]) {
  dft4(v[0], v[1], v[2], v[3]);
}

template <>
__device__ __forceinline__ void dft<8>(float2 (&v)[8]) {
  constexpr float kR = 0.70710678119f;
  // two of four over the even and the odd inputs
  dft4(v[0], v[2], v[4], v[6]);
  dft4(v[1], v[3], v[5], v[7]);
  v[3] = make_float2(kR * (v[3].x + v[3].y), kR * (v[3].y - v[3].x));
  v[5] = mul_mi(v[5]);
  v[7] = make_float2(kR * (v[7].y - v[7].x), -kR * (v[7].x + v[7].y));
#pragma unroll
  for (int i = 0; i < 8; i += 2) dft2(v[i], v[i + 1]);
  // v[2 k], v[2 k + 1] hold bins k, k + 4
  const float2 t1 = v[1], t2 = v[2], t3 = v[3], t4 = v[4], t5 = v[5], t6 = v[6];
  v[1] = t2;
  v[2] = t4;
  v[3] = t6;
  v[4] = t1;
  v[5] = t3;
  v[6] = t5;
}

// R = 4 Q: Q transforms of four over v[Q p + q], twiddles e^{-2 pi i q p'/R},
// four transforms of Q.
template <>
__device__ __forceinline__ void dft<16>(float2 (&v)[16]) {
  constexpr float kC = 0.92387953251f, kS = 0.38268343236f;
  constexpr float kR = 0.70710678119f;
#pragma unroll
  for (int q = 0; q < 4; ++q) dft4(v[q], v[4 + q], v[8 + q], v[12 + q]);
  // v[4 p' + q] times w16^(q p')
  v[5] = cmul(v[5], make_float2(kC, -kS));
  v[6] = cmul(v[6], make_float2(kR, -kR));
  v[7] = cmul(v[7], make_float2(kS, -kC));
  v[9] = cmul(v[9], make_float2(kR, -kR));
  v[10] = mul_mi(v[10]);
  v[11] = cmul(v[11], make_float2(-kR, -kR));
  v[13] = cmul(v[13], make_float2(kS, -kC));
  v[14] = cmul(v[14], make_float2(-kR, -kR));
  v[15] = cmul(v[15], make_float2(-kC, kS));
#pragma unroll
  for (int p = 0; p < 4; ++p)
    dft4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
  // v[4 p' + q'] is bin p' + 4 q': transpose
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < p; ++q) {
      const float2 t = v[4 * p + q];
      v[4 * p + q] = v[4 * q + p];
      v[4 * q + p] = t;
    }
}

template <>
__device__ __forceinline__ void dft<12>(float2 (&v)[12]) {
  constexpr float kS = 0.86602540378f;
#pragma unroll
  for (int q = 0; q < 3; ++q) dft4(v[q], v[3 + q], v[6 + q], v[9 + q]);
  // v[3 p' + q] times w12^(q p')
  v[4] = cmul(v[4], make_float2(kS, -0.5f));
  v[5] = cmul(v[5], make_float2(0.5f, -kS));
  v[7] = cmul(v[7], make_float2(0.5f, -kS));
  v[8] = cmul(v[8], make_float2(-0.5f, -kS));
  v[10] = mul_mi(v[10]);
  v[11] = make_float2(-v[11].x, -v[11].y);
#pragma unroll
  for (int p = 0; p < 4; ++p) dft3(v[3 * p], v[3 * p + 1], v[3 * p + 2]);
  // v[3 p' + q'] is bin p' + 4 q'
  float2 t[12];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int q = 0; q < 3; ++q) t[p + 4 * q] = v[3 * p + q];
#pragma unroll
  for (int i = 0; i < 12; ++i) v[i] = t[i];
}

// one word of padding per 16 keeps the strided stores of a pass on
// different banks
__device__ __forceinline__ int fft_pad(int i) { return i + (i >> 4); }

// One pass of the self-sorting (Stockham) transform of L points: radix R
// after passes of product NS.  load(i, r) gives input i (of the r-th share),
// the output goes to out.
template <int L, int R, int NS, int T, class Load>
__device__ __forceinline__ void fft_pass(Load load, float2 *out,
                                         const float2 *__restrict__ tw) {
#pragma unroll 1
  for (int i = threadIdx.x; i < L / R; i += T) {
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = load(i + r * (L / R), r);
    const int k = i % NS;
    if (NS > 1) {
      // w^r, w = e^{-2 pi i k / (NS R)} (tw: e^{-2 pi i n / (2 L)}): powers
      // of two from the table, the others as products of at most three
      constexpr int step = 2 * (L / (NS * R));
      float2 w[8];
#pragma unroll
      for (int r = 1; r < R && r < 8; ++r) {
        if ((r & (r - 1)) == 0) {
          w[r] = tw[(r * k) * step];
        } else {
          const int top = r >= 4 ? 4 : 2;
          w[r] = cmul(w[top], w[r - top]);
        }
        v[r] = cmul(v[r], w[r]);
      }
      if (R > 8) {
        const float2 w8 = tw[(8 * k) * step];
        v[8] = cmul(v[8], w8);
#pragma unroll
        for (int r = 9; r < R; ++r) v[r] = cmul(v[r], cmul(w8, w[r - 8]));
      }
    }
    dft<R>(v);
    const int o = (i / NS) * (NS * R) + k;
#pragma unroll
    for (int r = 0; r < R; ++r) out[fft_pad(o + r * NS)] = v[r];
  }
}

__host__ __device__ constexpr int fft_threads(int L) {
  return L <= 512 ? 64 : L <= 768 ? 96 : L <= 1024 ? 128 : L <= 1536 ? 192 : 256;
}
// at least 24 warps per SM (85 registers each)
__host__ __device__ constexpr int fft_min_ctas(int L) {
  return 768 / fft_threads(L);
}
// Y is carried times this beside X (X is Y's size times the cell number; 4
// keeps close pairs, a few cells from 0, and far ones at 1e-7)
constexpr int kFftScale = 4;

// What the CTAs that sum F(Q)'s partial histograms (fq_grid_reduce) need.
struct FqReduceArgs {
  HistRows rows;
  const KeyCols *keys;
  int n_keys, total;
  float *out;
};

// Gradient rows: CTA = (atom a of the part, in sorted order from a_first,
// coordinate).  X and Y of a
// row are the real and (negated) imaginary part of one real transform of
// length M = 2 L: of r_j = (y_j + s H_j)/2, r_{M-j} = (y_j - s H_j)/2 with
// y_j = j H_j, s = kFftScale, done as a complex transform of L points
// (c_n = r_2n + i r_2n+1) in three passes through shared memory.  The
// histogram parts of a unit are added as they are read, the cells below 0
// and above M/2 folded back.  Species of b are summed in registers with
// coef = -f_a f_b / na; bins below kbo are 0, NaN rows become 0.
// With F(Q) (gridDim.y 4) the first layer of CTAs sums its histograms beside
// the transforms: 20 us at 1,000 atoms that would else come after them.
// Bound by instruction issue (39 % of the slots at 16 warps per SM; 85
// registers leave room for 24): 30 ns per row of 1,500 bins over the GPU.
template <int R0, int R1, int R2>
__global__ void __launch_bounds__(fft_threads(R0 *R1 *R2),
                                  fft_min_ctas(R0 *R1 *R2))
    grad_transform_kernel(const float *__restrict__ rows,
                          const float *__restrict__ rows2,
                          const int *__restrict__ flag,
                          const int2 *__restrict__ parts,
                          const GradBlock *__restrict__ blocks, int n_species,
                          int a_first, const int *__restrict__ ext,
                          const int *__restrict__ perm,
                          const float2 *__restrict__ tw,
                          const float2 *__restrict__ pr,
                          const float *__restrict__ coef, int n_bins, int kbo,
                          float dq, float inv_bins, float *__restrict__ grad,
                          FqReduceArgs fr) {
  constexpr int L = R0 * R1 * R2, M = 2 * L, T = fft_threads(L);
  constexpr int KT = (L / 2 + T - 1) / T;  // bins per thread (K < L/2)
  extern __shared__ float2 fbuf[];
  float2 *b0 = fbuf, *b1 = fbuf + fft_pad(L);
  const int layers = gridDim.y - 3;
  if ((int)blockIdx.y < layers) {
    __shared__ int splan[32];
    const int per_key = fq_reduce_blocks(M, 8);
    for (int i = blockIdx.x; i < per_key * fr.n_keys; i += gridDim.x) {
      fq_grid_reduce(fr.rows, fr.keys[i / per_key], ext, 1, kGradPlan,
                     fr.total, M, i % per_key, 8, T / 8, fr.out + (size_t)(i / per_key) * fq_sum_floats(M),
                     reinterpret_cast<float *>(fbuf), splan);
      __syncthreads();
    }
    return;
  }
  const int words = grid_words(ext[0]), last = ext[0] + 4;
  const int ia = a_first + blockIdx.x, comp = blockIdx.y - layers;
  int sa = 0;  // (a species without atoms here starts where the next one does)
  while (sa + 1 < n_species && ia >= blocks[(sa + 1) * n_species].a0) ++sa;
  float acc[KT];
#pragma unroll
  for (int i = 0; i < KT; ++i) acc[i] = 0.f;
  for (int sb = 0; sb < n_species; ++sb) {
    const GradBlock B = blocks[sa * n_species + sb];
    if (B.cols == 0) continue;
    const int u = ia - B.a0;
    const int2 pw = parts[B.unit0 + u];
    const int slot0 = pw.x + B.unit0 + u, n_parts = pw.y - pw.x + 1;
    const float *h0 = rows + ((size_t)slot0 * 3 + comp) * words + kGridCell0;
    const float *g0 = rows2 + ((size_t)slot0 * 3 + comp) * words + kGridCell0;
    const size_t pstride = (size_t)3 * words;
    bool wide = false;
    for (int p = 0; p < n_parts; ++p) wide |= flag[slot0 + p] != 0;
    auto cell = [&](int j) {  // H_j
      float s = h0[j];
#pragma unroll 2
      for (int p = 1; p < n_parts; ++p) s += h0[p * pstride + j];
      return s;
    };
    auto cell2 = [&](int j) {  // n M w at j (only parts that have any)
      float s = 0.f;
      for (int p = 0; p < n_parts; ++p)
        if (flag[slot0 + p]) s += g0[p * pstride + j];
      return s;
    };
    __syncthreads();
    // (y_j, s H_j) / 2 of half a period; its two ends meet themselves
#pragma unroll 1
    for (int j = threadIdx.x; j <= L; j += T) {
      float y = 0.f, h = 0.f;
      if (j <= last) {
        h = cell(j);
        if (j >= 1 && j <= 3) h -= cell(-j);
        y = (float)j * h;
        if (wide) {
          y += cell2(j);
          if (j >= 1 && j <= 3) y += cell2(-j);
        }
      }
      if (j < L && M - j <= last) {
        const float x = cell(M - j);
        h -= x;
        y = fmaf((float)(M - j), x, y);
        if (wide) y += cell2(M - j);
      }
      b1[j] = j == 0 || j == L
                  ? make_float2(y, 0.f)
                  : make_float2(0.5f * y, (0.5f * kFftScale) * h);
    }
    __syncthreads();
    fft_pass<L, R0, 1, T>(
        [&](int n, int r) {
          // the upper half of the inputs mirrors the lower one
          if (2 * r < R0) {
            const float2 a = b1[2 * n], c = b1[2 * n + 1];
            return make_float2(a.x + a.y, c.x + c.y);
          }
          const float2 a = b1[M - 2 * n], c = b1[M - 2 * n - 1];
          return make_float2(a.x - a.y, c.x - c.y);
        },
        b0, tw);
    __syncthreads();
    fft_pass<L, R1, R0, T>([&](int n, int) { return b0[fft_pad(n)]; }, b1, tw);
    __syncthreads();
    fft_pass<L, R2, R0 * R1, T>([&](int n, int) { return b1[fft_pad(n)]; }, b0,
                                tw);
    __syncthreads();
    float near[kNearTerms];
    bool any = false;
#pragma unroll
    for (int n = 0; n < kNearTerms; ++n) {
      near[n] = 0.f;
      for (int p = 0; p < n_parts; ++p)
        near[n] += h0[p * pstride + n - kGridCell0];
      any |= near[n] != 0.f;
    }
    const float *cf = coef + ((size_t)sa * n_species + sb) * n_bins;
#pragma unroll
    for (int i = 0; i < KT; ++i) {
      const int k = threadIdx.x + i * T;
      if (k < kbo || k >= n_bins) continue;
      const float2 A = b0[fft_pad(k)], C = b0[fft_pad(k ? L - k : 0)];
      const float2 w = tw[k];  // (cos, -sin) of 2 pi k / M
      const float dr = A.x - C.x, di = A.y + C.y;
      const float X = 0.5f * (A.x + C.x + fmaf(w.x, di, w.y * dr));
      const float Y = (-0.5f / kFftScale) *
                      (A.y - C.y - fmaf(w.x, dr, -w.y * di));
      float g = fmaf(pr[k].x, X, -pr[k].y * Y);
      if (any) {
        // sum over near pairs of d (Q cos - sin/r)/r^2 = Q^3 sum_n (-1)^n
        // 2n/(2n+1)! (Q r)^(2n-2), n >= 1
        const float Q = (float)k * dq;
        const float z = -((float)k * inv_bins) * ((float)k * inv_bins);
        g -= Q * Q * Q *
             (near[0] * (1.f / 3.f) +
              z * (near[1] * (1.f / 30.f) +
                   z * (near[2] * (1.f / 840.f) +
                        z * (near[3] * (1.f / 45360.f) +
                             z * near[4] * (1.f / 3991680.f)))));
      }
      acc[i] = fmaf(cf[k], g, acc[i]);
    }
  }
  float *out = grad + ((size_t)perm[ia] * 3 + comp) * n_bins;
#pragma unroll
  for (int i = 0; i < KT; ++i) {
    const int k = threadIdx.x + i * T;
    if (k < n_bins) out[k] = k < kbo ? 0.f : nan_to_num_f(acc[i]);
  }
}

}  // namespace pyiid
