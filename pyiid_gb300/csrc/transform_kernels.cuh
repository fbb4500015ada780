// transform_kernels.cuh -- F(Q) -> G(r), potentials and the adjoint weights.
//
// The reference's F -> G transform (zero pad, odd extension, inverse FFT,
// linear interpolation onto the r grid) is a fixed linear map
//   G(r_i) = sum_k F_k T[k][i]
// (see the host builder of T for the derivation): get_pdf_at_qmin,
// fft_fq_to_gr and fft_gr_to_fq of pyiid/experiments/elasticscatter/
// kernels/master_kernel.py:39-203.  T is stored [n_bins][n_r]
// in FP32, so G for a batch of configurations is a skinny GEMM streaming T
// from HBM/L2 once per CTA column block.
#pragma once

#include <cooperative_groups.h>
#include <cstdint>
#include <cuda_runtime.h>

#include "adjoint_grid.cuh"

namespace pyiid {

// gr[b][i] = sum_k fq[b][k] * T[k][i]: FP32 products summed over blocks of
// 32 bins, the blocks in FP64 in their order.  CTA = (32 points r, NB
// configurations); the warps take the blocks of bins, so that a small batch
// still fills the GPU (one warp per 256 points and all bins took 30 us for
// one configuration of 330 x 4,000 against 9), and an element of T read from
// L2 serves NB configurations (64 of them: 35 us against 30, where the FP64
// sums of the blocks, 16 cycles an instruction, now take a third).
// Dynamic shared memory: blocks x NB x 32 partial sums.
constexpr int kPdfBlock = 32;  // bins
template <int NB>
__global__ void __launch_bounds__(512)
    pdf_kernel(const float *__restrict__ fq, const float *__restrict__ T,
               int n_bins, int n_r, int kmin, int n_configs,
               double *__restrict__ gr) {
  extern __shared__ float spart[];  // [block][NB][32]
  __shared__ float sf[16][kPdfBlock][NB];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_warps = blockDim.x >> 5;
  const int i = blockIdx.x * 32 + lane, b0 = blockIdx.y * NB;
  const int n_blocks = max(0, (n_bins - kmin + kPdfBlock - 1) / kPdfBlock);
  const float *Ti = T + min(i, n_r - 1);
  for (int blk = warp; blk < n_blocks; blk += n_warps) {
    const int k0 = kmin + blk * kPdfBlock, nk = min(kPdfBlock, n_bins - k0);
    __syncwarp();
#pragma unroll
    for (int b = 0; b < NB; ++b)
      sf[warp][lane][b] = lane < nk && b0 + b < n_configs
                              ? fq[(size_t)(b0 + b) * n_bins + k0 + lane]
                              : 0.f;
    __syncwarp();
    float part[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) part[b] = 0.f;
    if (nk == kPdfBlock) {
#pragma unroll 8
      for (int k = 0; k < kPdfBlock; ++k) {
        const float t = Ti[(size_t)(k0 + k) * n_r];
#pragma unroll
        for (int b = 0; b < NB; ++b)
          part[b] = fmaf(sf[warp][k][b], t, part[b]);
      }
    } else {
      for (int k = 0; k < nk; ++k) {
        const float t = Ti[(size_t)(k0 + k) * n_r];
#pragma unroll
        for (int b = 0; b < NB; ++b)
          part[b] = fmaf(sf[warp][k][b], t, part[b]);
      }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) spart[(blk * NB + b) * 32 + lane] = part[b];
  }
  __syncthreads();
  for (int b = warp; b < NB && b0 + b < n_configs; b += n_warps) {
    if (i >= n_r) break;
    double acc = 0.0;
    for (int blk = 0; blk < n_blocks; ++blk)
      acc += (double)spart[(blk * NB + b) * 32 + lane];
    gr[(size_t)(b0 + b) * n_r + i] = acc;
  }
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double *scratch) {
  // scratch: [32][NV]
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = warp_sum(v[i]);
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < NV; ++i) scratch[wid * NV + i] = v[i];
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double s = 0.0;
    for (int w = 0; w < nw; ++w) s += scratch[w * NV + i];
    v[i] = s;
  }
  __syncthreads();
}

// Potential per configuration, get_rw / get_chi_sq / get_scale
// of kernels/master_kernel.py:206-266, 388-389:
//   a = (gc.go)/(gc.gc); Rw: a <= 0 -> (1, 1), else sqrt(|go - a gc|^2/|go|^2)
//   chi^2: s = a if a > 0 else 1, value = |go - s gc|^2
// Optionally the adjoint vector c = d(value)/d(gcalc) exactly as the
// reference's get_grad_rw / get_grad_chi_sq contract it (the derivative of
// the scale uses the raw a even when the value used scale 1):
//   c_i = pre [s E_i + (gc.E) (go_i - 2 a gc_i)/(gc.gc)],  E = go - s gc,
//   pre = -Rw/|E|^2 (Rw) or -2 (chi^2).

// Sums over the 256 threads of every CTA of a cluster.  FP64 issues one warp
// instruction in 16 cycles here, so a warp per value adds what all threads
// have left in shared memory (13 instructions, against 5 in each of the
// eight warps by shuffles); the CTAs then read each other's sums there
// (distributed shared memory), in a fixed order.
struct ClusterSums {
  double part[4][256];
  double mine[4], total[4];
};
template <int NV>
__device__ __forceinline__ void cluster_sum(double (&v)[NV], ClusterSums &m) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) m.part[i][threadIdx.x] = v[i];
  __syncthreads();
  if (warp < NV) {
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += m.part[warp][32 * i + lane];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) m.mine[warp] = s;
  }
  cl.sync();
  if (warp < NV) {
    const int n = (int)cl.num_blocks();  // 1, 2 or 8
    double s = lane < n ? cl.map_shared_rank(m.mine, lane)[warp] : 0.0;
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) m.total[warp] = s;
  }
  cl.sync();  // nobody leaves, or writes again, before all have read
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = m.total[i];
}

// Potential of one configuration per cluster of CTAs, which share the points
// r: get_rw / get_chi_sq with get_scale as above.  FP64 bound; one CTA spent
// 39 us on 4,000 points, eight spend 11.
// weight (Rw only, may be null): per-point weights of get_rw
// (master_kernel.py:226-235): Rw = sqrt(sum w (go - a gc)^2 / sum w go^2)
// with the unweighted scale a; ee and gce (used by the gradients, which the
// reference never weights) stay unweighted.
__global__ void __launch_bounds__(256)
    potential_kernel(const double *__restrict__ gobs,
                     const double *__restrict__ gcalc, int n_r, int potential,
                     int ctas, double *__restrict__ out,
                     float *__restrict__ cvec,
                     const double *__restrict__ weight) {
  __shared__ ClusterSums sums;
  const int b = blockIdx.x / ctas;
  const int first = (blockIdx.x % ctas) * blockDim.x + threadIdx.x;
  const int step = ctas * blockDim.x;
  const double *gc = gcalc + (size_t)b * n_r;
  double v3[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = first; i < n_r; i += step) {
    const double c = gc[i], o = gobs[i];
    v3[0] += c * o;
    v3[1] += c * c;
    v3[2] += o * o;
    if (weight) v3[3] += weight[i] * o * o;
  }
  cluster_sum<4>(v3, sums);
  const double gco = v3[0], gcc = v3[1];
  const double goo = weight ? v3[3] : v3[2];
  const double a = gco / gcc;
  // the reference replaces a non-positive scale by 1; a NaN scale stays NaN
  const double s = (a <= 0.0) ? 1.0 : a;
  double v2[3] = {0.0, 0.0, 0.0};
  for (int i = first; i < n_r; i += step) {
    const double e = gobs[i] - s * gc[i];
    v2[0] += e * e;
    v2[1] += gc[i] * e;
    if (weight) v2[2] += weight[i] * e * e;
  }
  cluster_sum<3>(v2, sums);
  const double ee = v2[0], gce = v2[1];
  const double top = weight ? v2[2] : v2[0];
  const double value =
      potential == 0 ? (a <= 0.0 ? 1.0 : sqrt(top / goo)) : ee;
  if (first == 0) {
    out[2 * b] = value;
    out[2 * b + 1] = s;
  }
  if (cvec) {
    const double pre = (potential == 0) ? -value / ee : -2.0;
    const double ratio = gce / gcc;
    for (int i = first; i < n_r; i += step) {
      const double e = gobs[i] - s * gc[i];
      cvec[(size_t)b * n_r + i] =
          (float)(pre * (s * e + ratio * (gobs[i] - 2.0 * a * gc[i])));
    }
  }
}

// w[b][k] = sum_i T[k][i] c[b][i] in FP64 from FP32 lane sums, and with wk
// the weights of the pair-force tables (adjoint_grid.cuh) that follow from
// it.  CTA = NK bins x NB configurations: an element of T and one of c read
// serve NB and NK products (64 configurations of 330 x 4,000: 43 us with a
// warp per bin and configuration, 24 so), and one configuration still has a
// CTA per bin (19 us against 10).
template <int NK, int NB>
__global__ void __launch_bounds__(128)
    wvec_kernel(const float *__restrict__ T, const float *__restrict__ cvec,
                int n_bins, int n_r, int kmin, int n_configs,
                double *__restrict__ w, WkArgs wa) {
  __shared__ float red[NK * NB][129];
  const int k0 = blockIdx.x * NK, b0 = blockIdx.y * NB;
  float acc[NK][NB];
#pragma unroll
  for (int k = 0; k < NK; ++k)
#pragma unroll
    for (int b = 0; b < NB; ++b) acc[k][b] = 0.f;
  if (k0 + NK > kmin) {
#pragma unroll(NK * NB > 1 ? 2 : 8)
    for (int i = threadIdx.x; i < n_r; i += 128) {
      float t[NK], c[NB];
#pragma unroll
      for (int k = 0; k < NK; ++k)
        t[k] = T[(size_t)min(k0 + k, n_bins - 1) * n_r + i];
#pragma unroll
      for (int b = 0; b < NB; ++b)
        c[b] = cvec[(size_t)min(b0 + b, n_configs - 1) * n_r + i];
#pragma unroll
      for (int k = 0; k < NK; ++k)
#pragma unroll
        for (int b = 0; b < NB; ++b) acc[k][b] = fmaf(t[k], c[b], acc[k][b]);
    }
  }
#pragma unroll
  for (int k = 0; k < NK; ++k)
#pragma unroll
    for (int b = 0; b < NB; ++b) red[k * NB + b][threadIdx.x] = acc[k][b];
  __syncthreads();
  // 128 / (NK NB) threads per value (all of a warp at most) add fours of
  // lane sums in FP32, these in FP64
  constexpr int P = 128 / (NK * NB) > 32 ? 32 : 128 / (NK * NB);
  const int v = threadIdx.x / P, p = threadIdx.x % P;
  if (v >= NK * NB) return;  // whole warps
  double sum = 0.0;
  for (int i = p; i < 32; i += P)
    sum += (double)((red[v][i] + red[v][i + 32]) +
                    (red[v][i + 64] + red[v][i + 96]));
  for (int o = P / 2; o > 0; o >>= 1)
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const int k = k0 + v / NB, b = b0 + v % NB;
  if (p != 0 || k >= n_bins || b >= n_configs) return;
  if (k < kmin) sum = 0.0;
  w[(size_t)b * n_bins + k] = sum;
  if (wa.wk) adjoint_grid_weights(wa, b, k, k >= kmin, n_bins, sum);
}

// Adjoint tables: tabs[b][sa][sb][m] = (A_kk, A_kk+1, B_kk, B_kk+1),
//   kk = 2m, k = kb0 + kk, W = 2 w_k f_sa f_sb / na_k (0 outside
//   [kmin, n_bins) or where na_k = 0), A = k W, B = W.
__global__ void adjoint_table_kernel(const double *__restrict__ w,
                                     const double *__restrict__ na,
                                     const float *__restrict__ ftab,
                                     int n_species, int n_bins, int kmin,
                                     int kb0, int kp, int n_configs,
                                     float4 *__restrict__ tabs) {
  const int kh = kp / 2;
  const size_t total = (size_t)n_configs * n_species * n_species * kh;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int m = idx % kh;
    size_t rest = idx / kh;
    const int sb = rest % n_species;
    rest /= n_species;
    const int sa = rest % n_species;
    const int b = (int)(rest / n_species);
    float A[2], B[2];
    for (int e = 0; e < 2; ++e) {
      const int k = kb0 + 2 * m + e;
      double W = 0.0;
      if (k >= kmin && k < n_bins) {
        const double nak = na[(size_t)b * n_bins + k];
        if (nak != 0.0)
          W = 2.0 * w[(size_t)b * n_bins + k] * (double)ftab[sa * n_bins + k] *
              (double)ftab[sb * n_bins + k] / nak;
      }
      A[e] = (float)((double)k * W);
      B[e] = (float)W;
    }
    tabs[(((size_t)b * n_species + sa) * n_species + sb) * kh + m] =
        make_float4(A[0], A[1], B[0], B[1]);
  }
}

// dF coefficient table for the reference-convention gradient:
//   coef[b][sa][sb][k] = -f_sa f_sb / na_k   (float division as the reference)
__global__ void gradfq_coef_kernel(const double *__restrict__ na,
                                   const float *__restrict__ ftab,
                                   int n_species, int n_bins, int n_configs,
                                   float *__restrict__ coef) {
  const size_t total = (size_t)n_configs * n_species * n_species * n_bins;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    const int k = idx % n_bins;
    size_t rest = idx / n_bins;
    const int sb = rest % n_species;
    rest /= n_species;
    const int sa = rest % n_species;
    const int b = (int)(rest / n_species);
    const float nak = (float)na[(size_t)b * n_bins + k];
    coef[idx] = -(ftab[sa * n_bins + k] * ftab[sb * n_bins + k]) / nak;
  }
}

// Compat potential gradient from an explicit grad_pdf: one warp per row,
// grad[row] = sum_i c_i gpdf[row][i], with c recomputed from (gcalc, gobs).
__global__ void potential_grad_rows_kernel(const double *__restrict__ gpdf,
                                           const float *__restrict__ cvec,
                                           int n_rows, int n_r,
                                           double *__restrict__ grad) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= n_rows) return;
  const double *row = gpdf + (size_t)gw * n_r;
  double acc = 0.0;
  for (int i = lane; i < n_r; i += 32) acc += (double)cvec[i] * row[i];
  acc = warp_sum(acc);
  if (lane == 0) grad[gw] = acc;
}

}  // namespace pyiid
