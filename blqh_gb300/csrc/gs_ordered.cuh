// The Lanczos step after the SpMV for real sectors: three-term update and one
// classical Gram-Schmidt pass against every stored vector, in a fixed order of
// operations. On the square torus the sectors (J, K) in {0, nphi/2}^2 can have an
// exactly twofold degenerate ground state (a two-dimensional representation of its
// fourfold rotations), and the vector a run returns is then decided by its
// rounding. So the order of every sum is part of the result here: tiles of GS_ROWS
// rows, one warp per (tile, vector) with lane t taking rows t, t + 32, ...;
// partials summed 256 at a time by warps, then over the warps; the correction
// summed over even and odd vectors. (The products keep one order up to 2^15 rows;
// beyond, the tuner's choice of their form is another one.) Complex sectors, where no
// such degeneracy has been met, take the fixed-point pass of gs_fixed.cuh, which is
// faster and reproducible too. (Complex sectors without room for its planes, with
// accumulate = 1 or with BLQH_GS_FP64=1, come here.)
//
// FP64-valued runs take FP64 dots (FP64 pipe); FP32-valued runs with double-float
// accumulation take double-float dots on FP32 planes kept next to each FP64
// Krylov vector V_k: Vh_k = the leading 24 bits (truncated), Vl_k = the rest
// rounded (Vh + Vl = V_k to 2^-48): error <= ~2^-46 sum |V_k| |w|, 8 bytes per
// entry at HBM speed. The correction sum_k h_k V_k (every |h_k| <= 2^-30 |w|,
// checked per step, else FP64) is summed in FP32 from Vh (4 bytes per entry).
//
// What bounds a step: small sectors the chain of dependent reads and launches,
// large ones the FP64 pipe (FP64 dots) or HBM. So the vectors are split over
// blocks (a small sector has few tiles: 5,940 rows are 6 tiles), reductions end in
// the kernel that consumes them or, for the dots, in the group's last block, and
// the six kernels of a step are chained by programmatic stream serialization.
// Measured per step without the SpMV (200 steps, one GB300): 5,940 rows
// 88 -> 30 us, 647,079 rows FP32 values 219 -> 187 us, FP64 values
// 358 -> 223 us.
#pragma once

#include "gs_fixed.cuh"

constexpr int GS_ROWS = 1024;

// Sum of p[0..n), 256 threads, in the fixed order: thread t sums p[t], p[t + 256],
// ..., then the block (valid in thread 0). Up to 32 values need the first warp only.
__device__ __forceinline__ double ordered_sum(const double* p, int64_t step, int n, double* red) {
  double a = 0;
  if (n <= 32) {
    if (threadIdx.x < 32) {
      if ((int)threadIdx.x < n) a += __ldcg(p + threadIdx.x * step);
      a = warp_sum(a);
    }
    return a;
  }
  for (int t = threadIdx.x; t < n; t += 256) a += __ldcg(p + t * step);
  return block_sum_256(a, red);
}

// The same sum by one warp (valid in every lane).
__device__ __forceinline__ double ordered_sum_warp(const double* p, int64_t step, int n) {
  double s = 0;
  for (int g = 0; g < 8 && g * 32 < n; g++) {
    double a = 0;
    for (int t = g * 32 + (int)(threadIdx.x & 31); t < n; t += 256) a += __ldcg(p + t * step);
    s += warp_sum(a);
  }
  return s;
}

// part[tile] = conj(V_j) w over the tile (re, im), w after the SpMV. One warp per tile.
template <bool CPLX>
__global__ void __launch_bounds__(32) k_alpha_o(const double* vj, const double* w, int64_t dim, double* part, Scal S) {
  pdl_begin();
  const int64_t r0 = (int64_t)blockIdx.x * GS_ROWS;
  const int nr = (int)(dim - r0 < GS_ROWS ? dim - r0 : GS_ROWS);
  const int stop = S.flags[0];
  double sr = 0, si = 0;
  if (CPLX) {
    const double2* v2 = reinterpret_cast<const double2*>(vj) + r0;
    const double2* w2 = reinterpret_cast<const double2*>(w) + r0;
    for (int t = threadIdx.x; t < nr; t += 32) {
      const double2 a = v2[t], b = w2[t];
      sr += a.x * b.x + a.y * b.y;
      si += a.x * b.y - a.y * b.x;
    }
  } else {
#pragma unroll 16
    for (int t = threadIdx.x; t < nr; t += 32) sr += vj[r0 + t] * w[r0 + t];
  }
  if (stop) return;
  sr = warp_sum(sr);
  if (CPLX) si = warp_sum(si);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = sr;
    part[2 * blockIdx.x + 1] = si;
  }
}

// Three-term step: w -= h_j V_j (the SpMV removed beta_j v_{j-1}), partials of
// |w|^2 per 256 EPT entries. EPT = 4 (four consecutive entries per thread) in the
// runs with double-float planes, else 1. Every block sums h_j itself, so large
// sectors take a few blocks per SM with several groups of entries each (2,528
// blocks at 647,079 rows: 25 us, 608: 18 us). pmax (complex): the group's largest
// high word of |w|, for the fixed-point product's scale, or null.
template <bool CPLX, int EPT>
__global__ void __launch_bounds__(256) k_local_o(const double* vj, double* w, int64_t dim, const double* apart,
                                                 int ntile, double* pnorm, unsigned* pmax, int ngroups, Scal S,
                                                 int j) {
  pdl_begin();
  static_assert(!CPLX || EPT == 1, "complex rows one per thread");
  __shared__ double red[8];
  __shared__ unsigned ured[8];
  __shared__ double s_h[2];
  const int stop = S.flags[0];
  double a[EPT], b[EPT], v[EPT], u[EPT];
  auto load = [&](int64_t i0) {
#pragma unroll
    for (int q = 0; q < EPT; q++) {
      const int64_t i = i0 + q;
      a[q] = b[q] = v[q] = u[q] = 0.0;
      if (i < dim) {
        if (CPLX) {
          const double2 x = reinterpret_cast<const double2*>(w)[i], y = reinterpret_cast<const double2*>(vj)[i];
          a[q] = x.x;
          b[q] = x.y;
          v[q] = y.x;
          u[q] = y.y;
        } else {
          a[q] = w[i];
          v[q] = vj[i];
        }
      }
    }
  };
  load(((int64_t)blockIdx.x * 256 + threadIdx.x) * EPT);
  if (stop) return;
  const double hr_ = ordered_sum(apart, 2, ntile, red);
  const double hi_ = CPLX ? ordered_sum(apart + 1, 2, ntile, red) : 0.0;
  if (threadIdx.x == 0) {
    s_h[0] = hr_;
    s_h[1] = hi_;
    if (blockIdx.x == 0) {
      S.alpha[j] = hr_;
      S.flags[4] = 0;
    }
  }
  __syncthreads();
  const double hr = s_h[0], hi = s_h[1];
  for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
    const int64_t i0 = ((int64_t)g * 256 + threadIdx.x) * EPT;
    if (g != (int)blockIdx.x) load(i0);
    double nn = 0;
    unsigned hw = 0;
#pragma unroll
    for (int q = 0; q < EPT; q++) {
      const int64_t i = i0 + q;
      if (i < dim) {
        if (CPLX) {
          a[q] -= hr * v[q] - hi * u[q];
          b[q] -= hr * u[q] + hi * v[q];
          reinterpret_cast<double2*>(w)[i] = make_double2(a[q], b[q]);
          nn += a[q] * a[q] + b[q] * b[q];
          hw = max(abs_high_word(a[q]), abs_high_word(b[q]));
        } else {
          a[q] -= hr * v[q];
          w[i] = a[q];
          nn += a[q] * a[q];
        }
      }
    }
    nn = block_sum_256(nn, red);
    if (threadIdx.x == 0) pnorm[g] = nn;
    if (CPLX && pmax) {
      hw = block_max(hw, ured);
      if (threadIdx.x == 0) pmax[g] = hw;
      __syncthreads();  // ured is written again
    }
  }
}

// (ah, al) += (vh + vl) (wh + wl) in double-float (the vl wl term, ~2^-48 of the
// product, is dropped).
__device__ __forceinline__ void df_prod_split(float& ah, float& al, float vh, float vl, float wh, float wl) {
  const float p = vh * wh;
  const float pe = fmaf(vh, wh, -p);
  const float t = fmaf(vh, wl, fmaf(vl, wh, pe));
  float s, e;
  two_sum(ah, p, s, e);
  ah = s;
  al += e + t;
}

// The warp's sums of four values at once, in the order warp_sum adds them: after
// the first level the two half-warps carry two values, after the second the four
// quarters carry four, so that four sums take 6 FP64 additions instead of 20. The
// sum of value q ends in lanes 8 q .. 8 q + 7 (q = 2 b16 + b8 of the lane).
__device__ __forceinline__ double warp_sum4(double s0, double s1, double s2, double s3) {
  const int lane = threadIdx.x & 31;
  const bool hi16 = lane & 16, hi8 = lane & 8;
  // lanes below 16 keep s0 and s1, the others s2 and s3
  double a = hi16 ? s2 : s0, b = hi16 ? s3 : s1;
  a += __shfl_xor_sync(0xffffffffu, hi16 ? s0 : s2, 16);
  b += __shfl_xor_sync(0xffffffffu, hi16 ? s1 : s3, 16);
  double c = hi8 ? b : a;
  c += __shfl_xor_sync(0xffffffffu, hi8 ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  return c;
}

// Full pass, dots: h2[k] = conj(V_k) w for k in [0, nk). A block takes one tile
// (w's tile in shared memory) and gk vectors, one warp per KB vectors at a time
// (KB = 4 for the FP64 dots of large real sectors: four chains hide the pipe's
// latency and share warp_sum4 and the reads of w; 182 -> 137 us at 647,079 rows
// and 100 vectors, 16 blocks per SM instead of 4 included); gk
// is 8 where the tiles are few and grows until the blocks fill the GPU four times,
// so that large sectors stage w's tile once. DF: from the planes (row stride ld),
// 16-byte loads. With `finish` (few tiles) the last block of a group sums its
// vectors' partials (part[k][tile]) and sets flags[4] when a coefficient is not
// below 2^-30 |w|; else k_reduce_o does, one block per vector (where the line lies:
// gs_step_o).
template <bool CPLX, bool DF, int KB>
__global__ void __launch_bounds__(256) k_dots_o(const double* V, const float* Vh, const float* Vl, int64_t ld,
                                                int64_t dim, int ntile, int nk, int gk, int ngroups, const double* w,
                                                double* part, const double* pnorm, int npn, int finish, Scal S,
                                                int j) {
  pdl_begin();
  static_assert(!CPLX || !DF, "complex sectors without the fixed-point planes use FP64");
  static_assert(KB == 1 || (KB == 4 && !CPLX && !DF), "four vectors per warp: real FP64");
  constexpr int VW = CPLX ? 2 : 1;
  constexpr int TF = GS_ROWS * VW;
  __shared__ __align__(16) double ws[TF];  // DF: the (hi, lo) planes of w's tile
  __shared__ double red[8];
  __shared__ double s_nrm;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int tile = (int)(blockIdx.x / (unsigned)ngroups), g = (int)(blockIdx.x % (unsigned)ngroups);
  const int ka = g * gk, kb = min(nk, ka + gk);
  const int64_t r0 = (int64_t)tile * GS_ROWS;
  const int nr = (int)(dim - r0 < GS_ROWS ? dim - r0 : GS_ROWS);
  const int stop = S.flags[0];
  float* wh = reinterpret_cast<float*>(ws);
  float* wl = wh + GS_ROWS;
#pragma unroll 4
  for (int t = threadIdx.x; t < TF; t += 256) {
    const double x = t < nr * VW ? w[r0 * VW + t] : 0.0;
    if (DF) {
      const float2 p = split_f64(x);
      wh[t] = p.x;
      wl[t] = p.y;
    } else {
      ws[t] = x;
    }
  }
  if (stop) return;
  __syncthreads();
  if (KB == 4) {
    for (int k = ka + wid * 4; k < kb; k += 32) {
      const double* vk[4];
#pragma unroll
      for (int b = 0; b < 4; b++) vk[b] = V + (int64_t)min(k + b, kb - 1) * dim + r0;  // past the end: the last again
      double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
      for (int t = lane; t < nr; t += 32) {
        const double x = ws[t];
#pragma unroll
        for (int b = 0; b < 4; b++) s[b] += vk[b][t] * x;
      }
      const double r = warp_sum4(s[0], s[1], s[2], s[3]);
      const int b = lane >> 3;
      if ((lane & 7) == 0 && k + b < kb) part[(int64_t)(k + b) * ntile + tile] = r;
    }
  }
  for (int k = ka + wid; KB == 1 && k < kb; k += 8) {
    if (DF) {
      const float* ph = Vh + (int64_t)k * ld + r0;
      const float* pl = Vl + (int64_t)k * ld + r0;
      float sh = 0.f, sl = 0.f;
#pragma unroll 2
      for (int t = lane * 4; t < nr; t += 128) {  // the row padding keeps t + 3 inside the plane
        const float4 h4 = __ldcs(reinterpret_cast<const float4*>(ph + t));
        const float4 l4 = __ldcs(reinterpret_cast<const float4*>(pl + t));
        const float4 a4 = *reinterpret_cast<const float4*>(wh + t);
        const float4 b4 = *reinterpret_cast<const float4*>(wl + t);
        df_prod_split(sh, sl, h4.x, l4.x, a4.x, b4.x);
        df_prod_split(sh, sl, h4.y, l4.y, a4.y, b4.y);
        df_prod_split(sh, sl, h4.z, l4.z, a4.z, b4.z);
        df_prod_split(sh, sl, h4.w, l4.w, a4.w, b4.w);
      }
      df_seg_reduce<32>(sh, sl);
      if (lane == 0) part[(int64_t)k * ntile + tile] = (double)sh + (double)sl;
    } else {
      const double* vk = V + ((int64_t)k * dim + r0) * VW;
      double sr = 0, si = 0;
      if (CPLX) {
        for (int t = lane; t < nr; t += 32) {
          const double2 a = reinterpret_cast<const double2*>(vk)[t];
          const double br = ws[2 * t], bi = ws[2 * t + 1];
          sr += a.x * br + a.y * bi;
          si += a.x * bi - a.y * br;
        }
      } else {
#pragma unroll 8
        for (int t = lane; t < nr; t += 32) sr += vk[t] * ws[t];
      }
      sr = warp_sum(sr);
      if (CPLX) si = warp_sum(si);
      if (lane == 0) {
        part[((int64_t)k * ntile + tile) * VW] = sr;
        if (CPLX) part[((int64_t)k * ntile + tile) * VW + 1] = si;
      }
    }
  }
  if (!finish || !last_block(S.cnt + CNT_DOTS + g, ntile)) return;
  const double nrm = ordered_sum(pnorm, 1, npn, red);
  if (threadIdx.x == 0) s_nrm = nrm;
  __syncthreads();
  for (int k = ka + wid; k < kb; k += 8) {
    const double* p = part + (int64_t)k * ntile * VW;
    const double a = ordered_sum_warp(p, VW, ntile);
    const double b = CPLX ? ordered_sum_warp(p + 1, VW, ntile) : 0.0;
    if (lane == 0) {
      S.h2[2 * k] = a;
      S.h2[2 * k + 1] = b;
      // the correction is summed in FP32 only while every coefficient is below 2^-30 |w|
      if (a * a + b * b > 0x1p-60 * s_nrm) atomicOr(S.flags + 4, 1);
      if (k == j) S.alpha[j] += a;
    }
  }
}

// The dots' partials of vector blockIdx.x summed (see k_dots_o).
template <bool CPLX>
__global__ void __launch_bounds__(256) k_reduce_o(const double* part, int ntile, const double* pnorm, int npn, Scal S,
                                                  int j) {
  pdl_begin();
  if (S.flags[0]) return;
  __shared__ double red[8];
  constexpr int VW = CPLX ? 2 : 1;
  const int k = blockIdx.x;
  const double* p = part + (int64_t)k * ntile * VW;
  const double a = ordered_sum(p, VW, ntile, red);
  const double b = CPLX ? ordered_sum(p + 1, VW, ntile, red) : 0.0;
  const double nrm = ordered_sum(pnorm, 1, npn, red);
  if (threadIdx.x != 0) return;
  S.h2[2 * k] = a;
  S.h2[2 * k + 1] = b;
  // the correction is summed in FP32 only while every coefficient is below 2^-30 |w|
  if (a * a + b * b > 0x1p-60 * nrm) atomicOr(S.flags + 4, 1);
  if (k == j) S.alpha[j] += a;
}

// Full pass, correction: w -= sum_k h2[k] V_k, partials of |w|^2 (and pmax) as in k_local_o.
// In FP32 from FP32-truncated coefficients and entries (the Vh plane where there
// is one, PL, else V truncated here; relative error ~2^-22 of a correction <=
// 2^-30 |w|, below FP64's rounding of w), subtracted in FP64. A flagged pass uses
// FP64 FMAs on V. BATCH vectors' loads are in flight per thread.
template <bool CPLX, int EPT, bool PL>
__global__ void __launch_bounds__(256) k_update_o(const double* V, const float* Vh, int64_t ld, int64_t dim, int nk,
                                                  double* w, double* pnorm, unsigned* pmax, Scal S) {
  pdl_begin();
  static_assert(!CPLX || (EPT == 1 && !PL), "complex rows one per thread, from V");
  __shared__ unsigned ured[8];
  if (S.flags[0]) return;
  extern __shared__ double hs[];  // [2 nk] coefficients, then [2 nk] floats
  __shared__ double red[8];
  float* hf = reinterpret_cast<float*>(hs + 2 * nk);
  const bool lowp = !S.flags[4];
  const int64_t i0 = ((int64_t)blockIdx.x * 256 + threadIdx.x) * EPT;
  double a[EPT], b = 0;
#pragma unroll
  for (int q = 0; q < EPT; q++) {
    a[q] = 0.0;
    if (i0 + q < dim) {
      if (CPLX) {
        const double2 x = reinterpret_cast<const double2*>(w)[i0 + q];
        a[q] = x.x;
        b = x.y;
      } else {
        a[q] = w[i0 + q];
      }
    }
  }
  for (int t = threadIdx.x; t < 2 * nk; t += 256) {
    const double c = S.h2[t];
    hs[t] = c;
    hf[t] = f64_lead_f32(c);
  }
  __syncthreads();
  double nn = 0;
  if (i0 < dim) {
    if (CPLX) {
      const double2* p = reinterpret_cast<const double2*>(V) + i0;
      if (lowp) {
        float dr = 0.f, di = 0.f;
        for (int k = 0; k < nk; k++) {
          const double2 v = p[(int64_t)k * dim];
          const float vr = f64_lead_f32(v.x), vi = f64_lead_f32(v.y);
          const float hr = hf[2 * k], hi = hf[2 * k + 1];
          dr = fmaf(hr, vr, fmaf(-hi, vi, dr));
          di = fmaf(hr, vi, fmaf(hi, vr, di));
        }
        a[0] -= (double)dr;
        b -= (double)di;
      } else {
        for (int k = 0; k < nk; k++) {
          const double2 v = p[(int64_t)k * dim];
          const double hr = hs[2 * k], hi = hs[2 * k + 1];
          a[0] -= hr * v.x - hi * v.y;
          b -= hr * v.y + hi * v.x;
        }
      }
      reinterpret_cast<double2*>(w)[i0] = make_double2(a[0], b);
      nn = a[0] * a[0] + b * b;
    } else {
      if (lowp) {
        float d0[EPT], d1[EPT];  // even and odd k
#pragma unroll
        for (int q = 0; q < EPT; q++) d0[q] = d1[q] = 0.f;
        constexpr int BATCH = EPT == 4 ? 8 : 32;
        auto load = [&](float (&x)[EPT], int k) {
          if (EPT == 4) {
            const float4 v = __ldcs(reinterpret_cast<const float4*>(Vh + (int64_t)k * ld + i0));
            x[0] = v.x;
            x[EPT / 4] = v.y;  // indices 1, 2, 3 for EPT = 4
            x[EPT / 2] = v.z;
            x[EPT - 1] = v.w;
          } else {
            x[0] = PL ? __ldcs(Vh + (int64_t)k * ld + i0) : f64_lead_f32(V[(int64_t)k * dim + i0]);
          }
        };
        int k = 0;
        for (; k + BATCH <= nk; k += BATCH) {
          float x[BATCH][EPT];
#pragma unroll
          for (int u = 0; u < BATCH; u++) load(x[u], k + u);
#pragma unroll
          for (int u = 0; u < BATCH; u++)
#pragma unroll
            for (int q = 0; q < EPT; q++) {
              if (u & 1) d1[q] = fmaf(hf[2 * (k + u)], x[u][q], d1[q]);
              else d0[q] = fmaf(hf[2 * (k + u)], x[u][q], d0[q]);
            }
        }
        float x[BATCH][EPT];
#pragma unroll
        for (int u = 0; u < BATCH; u++)
          if (k + u < nk) load(x[u], k + u);
#pragma unroll
        for (int u = 0; u < BATCH; u++)
          if (k + u < nk)
#pragma unroll
            for (int q = 0; q < EPT; q++) {
              if (u & 1) d1[q] = fmaf(hf[2 * (k + u)], x[u][q], d1[q]);
              else d0[q] = fmaf(hf[2 * (k + u)], x[u][q], d0[q]);
            }
#pragma unroll
        for (int q = 0; q < EPT; q++) a[q] -= (double)(d0[q] + d1[q]);
      } else {
        for (int k = 0; k < nk; k++) {
          const double* vk = V + (int64_t)k * dim + i0;
          const double hr = hs[2 * k];
#pragma unroll
          for (int q = 0; q < EPT; q++)
            if (i0 + q < dim) a[q] -= hr * vk[q];
        }
      }
#pragma unroll
      for (int q = 0; q < EPT; q++)
        if (i0 + q < dim) {
          w[i0 + q] = a[q];
          nn += a[q] * a[q];
        }
    }
  }
  nn = block_sum_256(nn, red);
  if (threadIdx.x == 0) pnorm[blockIdx.x] = nn;
  if (CPLX && pmax) {
    const unsigned hw = block_max(max(abs_high_word(a[0]), abs_high_word(b)), ured);
    if (threadIdx.x == 0) pmax[blockIdx.x] = hw;
  }
}

// Where v_{j+1} goes: V, the SpMV's split input, the planes (rows padded with zeros to ld floats).
struct NextPlanes {
  double* v;
  float2* xs;
  int2* xq;
  int* xe;  // the exponent xq is below
  float* vh;
  float* vl;
  int64_t ld;
};

// v_{j+1} = w / beta_{j+1}, beta from the partials of |w|^2 and, for the fixed-point
// product, the scale of its input from pmax (taken together by every block, so there
// are few of them, grid-stride). start: src is the start vector, only its
// planes are written.
__global__ void __launch_bounds__(256) k_scale_o(const double* src, int64_t n, int start, const double* pnorm,
                                                 const unsigned* pmax, int npn, Scal S, int j, double breakdown_tol,
                                                 NextPlanes nx) {
  pdl_begin();
  if (S.flags[0]) return;
  __shared__ double red[8];
  __shared__ unsigned ured[8];
  __shared__ double s_inv;
  __shared__ int s_xe;
  if (!start) {
    const double s = ordered_sum(pnorm, 1, npn, red);
    unsigned hw = 0;
    if (nx.xq) {
      for (int t = threadIdx.x; t < npn; t += 256) hw = max(hw, __ldcg(pmax + t));
      hw = block_max(hw, ured);
    }
    if (threadIdx.x == 0) {
      s_inv = 1.0 / sqrt(s);
      if (nx.xq) {
        s_xe = scaled_exponent(word_exponent(hw), 0.0, s_inv);
        if (blockIdx.x == 0) *nx.xe = s_xe;
      }
      if (blockIdx.x == 0) beta_from(S, j, s, breakdown_tol);
    }
  }
  __syncthreads();
  const double inv = start ? 1.0 : s_inv;
  const int64_t end = nx.vh ? (nx.ld > n ? nx.ld : n) : n;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < end; i += (int64_t)gridDim.x * 256) {
    double v = 0.0;
    if (i < n) {
      v = src[i];
      if (!start) {
        v *= inv;
        store_entry(v, i, nx.v, nx.xs, nx.xq, s_xe);
      }
    }
    if (nx.vh) {
      const float h = f64_lead_f32(v);
      nx.vh[i] = h;
      if (nx.vl) nx.vl[i] = (float)(v - (double)h);
    }
  }
}
