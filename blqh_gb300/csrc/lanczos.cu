// K3 SpMV, K4/K5 Lanczos steps with full FP64 reorthogonalization, K6 the
// tridiagonal eigensolver, K7 the Ritz vector, and the Rayleigh quotients.
//
// Replaces Mat::operator* (BLQH_without_spin/matrix.cpp:244-267),
// lhamil::coeff_explicit_update (lanczos_hamiltonian.cpp:453-579), lhamil::diag
// with LAPACK dsyevd (lanczos_hamiltonian.cpp:581-606, matrix.cpp:288-305),
// eigenstates_reconstruction (:610-644) and ground_state_energy (:646-656).
//
// Differences by design (the physics answer is the same):
//   * the Krylov basis is kept in HBM, so the ground state is one GEMV over it
//     instead of a second Lanczos pass, and it is not complex-conjugated (the
//     reference's conjugated reconstruction is an eigenvector only in real
//     sectors);
//   * with reorth = 1 every new vector, after the three-term step, is
//     orthogonalized against all previous ones by one classical Gram-Schmidt
//     pass, so no ghost Ritz values appear and the run stops at convergence or
//     at an invariant subspace (dim < lambda);
//   * all scalars (alpha, beta, Gram-Schmidt coefficients, stop flag) stay in
//     device memory; the host polls the stop flag once per chunk of steps.
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cmath>
#include <cstring>

#include "../../include/blqh_gpu_debug.h"
#include "krylov.cuh"
#include "gs_ordered.cuh"
#include "sector.cuh"
#include "tridiag.cuh"

double rayleigh_regen_impl(blqh_ctx* ctx, const blqh_basis* B, const blqh_params& p, const double* d_psi,
                           bool want_complex);
void spin_observables_impl(blqh_ctx* ctx, const blqh_basis* B, const double* psi, int cplx, double* out);
double spin_rayleigh_regen_impl(blqh_ctx* ctx, const blqh_basis* B, const blqh_params_spin& p, const double* x);
int hamil_build_impl(blqh_ctx* ctx, const blqh_basis* B, const blqh_params& p, int prec, blqh_csr* M);
void free_csr(blqh_csr* m);
void debug_batch_pass(blqh_ctx* ctx, const double* V, double* w, int64_t N, int nk, double* h, bool update);

namespace {

// ---------------------------------------------------------------------------
// SpMV: LPR lanes per row, FP64 accumulation. y = H x - b * xprev.
template <class VT>
__device__ __forceinline__ double2 ld_val(const VT* v, int64_t k);
template <>
__device__ __forceinline__ double2 ld_val<double>(const double* v, int64_t k) {
  return make_double2(__ldg(v + k), 0.0);
}
template <>
__device__ __forceinline__ double2 ld_val<float>(const float* v, int64_t k) {
  return make_double2((double)__ldg(v + k), 0.0);
}
template <>
__device__ __forceinline__ double2 ld_val<double2>(const double2* v, int64_t k) {
  return __ldg(v + k);
}
template <>
__device__ __forceinline__ double2 ld_val<float2>(const float2* v, int64_t k) {
  float2 f = __ldg(v + k);
  return make_double2((double)f.x, (double)f.y);
}

template <class VT, bool CPLX, int LPR>
__global__ void __launch_bounds__(256) k_spmv(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                                              const VT* __restrict__ val, const double* __restrict__ x,
                                              double* __restrict__ y, int64_t dim, const double* bptr,
                                              const double* __restrict__ xprev, const int* stop) {
  if (stop && *stop) return;
  // warp-uniform iteration: every lane of a warp runs the same number of row
  // rounds, so the segmented shuffles below always see all 32 lanes.
  const int lane = threadIdx.x & 31;
  constexpr int GPW = 32 / LPR;  // rows per warp per round
  const int gi = lane / LPR, sub = lane % LPR;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const double b = bptr ? *bptr : 0.0;
  for (int64_t rb = warp * GPW; rb < dim; rb += nwarps * GPW) {
    const int64_t r = rb + gi;
    const bool ok = r < dim;
    const int64_t s = ok ? rp[r] : 0, e = ok ? rp[r + 1] : 0;
    double ar = 0.0, ai = 0.0;
    int64_t k = s + sub;
#pragma unroll 4
    for (; k < e; k += LPR) {
      const int32_t c = __ldg(col + k);
      const double2 v = ld_val<VT>(val, k);
      if (CPLX) {
        const double2 xv = __ldg(reinterpret_cast<const double2*>(x) + c);
        ar += v.x * xv.x - v.y * xv.y;
        ai += v.x * xv.y + v.y * xv.x;
      } else {
        ar += v.x * __ldg(x + c);
      }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) {
      ar += __shfl_xor_sync(0xffffffffu, ar, o, LPR);
      if (CPLX) ai += __shfl_xor_sync(0xffffffffu, ai, o, LPR);
    }
    if (ok && sub == 0) {
      if (CPLX) {
        double2 o = make_double2(ar, ai);
        if (xprev) {
          const double2 p = reinterpret_cast<const double2*>(xprev)[r];
          o.x -= b * p.x;
          o.y -= b * p.y;
        }
        reinterpret_cast<double2*>(y)[r] = o;
      } else {
        y[r] = xprev ? ar - b * xprev[r] : ar;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// SpMV with double-float accumulation for FP32-valued CSR (helpers in krylov.cuh).
template <bool CPLX, int LPR>
__global__ void __launch_bounds__(256) k_spmv_df(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                                                 const float* __restrict__ val, const float2* __restrict__ xs,
                                                 double* __restrict__ y, int64_t dim, const double* bptr,
                                                 const double* __restrict__ xprev, const int* stop) {
  if (stop && *stop) return;
  const int lane = threadIdx.x & 31;
  constexpr int GPW = 32 / LPR;
  const int gi = lane / LPR, sub = lane % LPR;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const double b = bptr ? *bptr : 0.0;
  for (int64_t rb = warp * GPW; rb < dim; rb += nwarps * GPW) {
    const int64_t r = rb + gi;
    const bool ok = r < dim;
    const int64_t s = ok ? rp[r] : 0, e = ok ? rp[r + 1] : 0;
    float rh = 0.f, rl = 0.f, ih = 0.f, il = 0.f;
#pragma unroll 4
    for (int64_t k = s + sub; k < e; k += LPR) {
      const int32_t c = __ldg(col + k);
      if (CPLX) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(val) + k);
        const float4 x = __ldg(reinterpret_cast<const float4*>(xs) + c);  // (re hi, re lo, im hi, im lo)
        df_add_prod(rh, rl, v.x, x.x, x.y);
        df_add_prod(rh, rl, -v.y, x.z, x.w);
        df_add_prod(ih, il, v.x, x.z, x.w);
        df_add_prod(ih, il, v.y, x.x, x.y);
      } else {
        const float v = __ldg(val + k);
        const float2 x = __ldg(xs + c);
        df_add_prod(rh, rl, v, x.x, x.y);
      }
    }
    df_seg_reduce<LPR>(rh, rl);
    if (CPLX) df_seg_reduce<LPR>(ih, il);
    if (ok && sub == 0) {
      const double re = (double)rh + (double)rl;
      if (CPLX) {
        double2 o = make_double2(re, (double)ih + (double)il);
        if (xprev) {
          const double2 p = reinterpret_cast<const double2*>(xprev)[r];
          o.x -= b * p.x;
          o.y -= b * p.y;
        }
        reinterpret_cast<double2*>(y)[r] = o;
      } else {
        y[r] = xprev ? re - b * xprev[r] : re;
      }
    }
  }
}

// Real FP32-valued CSR, double-float accumulation, 16-byte loads: each lane
// takes four consecutive nonzeros (one int4 of columns, one float4 of values)
// per step, so a warp keeps 512 B of matrix stream in flight per load pair and
// issues the four gathers of x back to back. The unaligned head (< 4 entries
// before a 16-byte boundary) and tail of each row are loaded one by one.
template <int LPR>
__global__ void __launch_bounds__(256) k_spmv_df_v4(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                                                    const float* __restrict__ val, const float2* __restrict__ xs,
                                                    double* __restrict__ y, int64_t dim, const double* bptr,
                                                    const double* __restrict__ xprev, const int* stop) {
  if (stop && *stop) return;
  const int lane = threadIdx.x & 31;
  constexpr int GPW = 32 / LPR;
  const int gi = lane / LPR, sub = lane % LPR;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  // Each warp takes chunks of 32 consecutive rows; lane k keeps the sum of row
  // base + k, and the FP64 epilogue runs once per chunk with all lanes busy
  // (an FP64 instruction costs the same with one active lane as with 32).
  for (int64_t base = warp * 32; base < dim; base += nwarps * 32) {
   float mh = 0.f, ml = 0.f;
   for (int rd = 0; rd < LPR; rd++) {
    const int64_t r = base + rd * GPW + gi;
    const bool ok = r < dim;
    const int64_t s = ok ? __ldg(rp + r) : 0, e = ok ? __ldg(rp + r + 1) : 0;
    float ah = 0.f, al = 0.f;
    const int64_t a4 = (s + 3) & ~(int64_t)3;   // first 16-byte aligned index
    const int64_t b4 = e & ~(int64_t)3;         // end of the aligned body
    const int64_t hend = a4 < e ? a4 : e;
    if (s + sub < hend) {
      const int64_t k = s + sub;
      const float2 x = __ldg(xs + __ldg(col + k));
      df_add_prod(ah, al, __ldg(val + k), x.x, x.y);
    }
    if (b4 > a4) {
      const int4* c4 = reinterpret_cast<const int4*>(col);
      const float4* v4 = reinterpret_cast<const float4*>(val);
      for (int64_t q = (a4 >> 2) + sub; q < (b4 >> 2); q += LPR) {
        const int4 c = __ldg(c4 + q);
        const float4 v = __ldg(v4 + q);
        const float2 x0 = __ldg(xs + c.x), x1 = __ldg(xs + c.y), x2 = __ldg(xs + c.z), x3 = __ldg(xs + c.w);
        df_add_prod(ah, al, v.x, x0.x, x0.y);
        df_add_prod(ah, al, v.y, x1.x, x1.y);
        df_add_prod(ah, al, v.z, x2.x, x2.y);
        df_add_prod(ah, al, v.w, x3.x, x3.y);
      }
      if (b4 + sub < e) {
        const int64_t k = b4 + sub;
        const float2 x = __ldg(xs + __ldg(col + k));
        df_add_prod(ah, al, __ldg(val + k), x.x, x.y);
      }
    }
    df_seg_reduce<LPR>(ah, al);
    // every lane of a segment holds its row's sum; lane k collects row base + k
    const int src = (lane % GPW) * LPR;
    const float th = __shfl_sync(0xffffffffu, ah, src), tl = __shfl_sync(0xffffffffu, al, src);
    if (lane / GPW == rd) {
      mh = th;
      ml = tl;
    }
   }
   const int64_t r = base + lane;
   if (r < dim) {
     const double re = (double)mh + (double)ml;
     y[r] = xprev ? re - *bptr * xprev[r] : re;
   }
  }
}

// x (FP64) -> (hi, lo) FP32 pairs for the double-float SpMV.
__global__ void k_split(const double* __restrict__ x, float2* __restrict__ xs, int64_t n, const int* stop) {
  if (stop && *stop) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double v = x[i];
    const float hi = (float)v;
    xs[i] = make_float2(hi, (float)(v - (double)hi));
  }
}

// ---------------------------------------------------------------------------
// <psi|H|psi> with each FP64 element carried as v32 + res (FP32 value and the
// FP32 rest of the builder's FP64 value, 2^-48 relative): y = H32 psi comes
// from the double-float SpMV; here one warp per row sums res * psi_hi in FP32
// (the rest is 2^-24 of the element, so FP32 keeps 2^-48 of the total) and
// adds Re(conj(psi_r) (y_r + that sum)) in FP64 into a block partial. Rows go
// to warps in a fixed grid-stride order: the result is reproducible.
template <bool CPLX>
__global__ void __launch_bounds__(256) k_rq_res(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                                                const void* __restrict__ res, const float2* __restrict__ xs,
                                                const double* __restrict__ psi, const double* __restrict__ y,
                                                int64_t dim, double* __restrict__ part) {
  __shared__ double red[8];
  const int lane = threadIdx.x & 31;
  const int64_t wg = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  double acc = 0;
  for (int64_t r = wg; r < dim; r += nw) {
    const int64_t a = rp[r], e = rp[r + 1];
    float sr = 0.f, si = 0.f;
    for (int64_t k = a + lane; k < e; k += 32) {
      const int c = __ldg(col + k);
      if (CPLX) {
        const float2 rv = __ldg(reinterpret_cast<const float2*>(res) + k);
        const float4 x = __ldg(reinterpret_cast<const float4*>(xs) + c);  // (re hi, re lo, im hi, im lo)
        sr = fmaf(rv.x, x.x, fmaf(-rv.y, x.z, sr));
        si = fmaf(rv.x, x.z, fmaf(rv.y, x.x, si));
      } else {
        sr = fmaf(__ldg(reinterpret_cast<const float*>(res) + k), __ldg(xs + c).x, sr);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      if (CPLX) si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (lane == 0) {
      if (CPLX) acc += psi[2 * r] * (y[2 * r] + (double)sr) + psi[2 * r + 1] * (y[2 * r + 1] + (double)si);
      else acc += psi[r] * (y[r] + (double)sr);
    }
  }
  const double t = block_sum_256(acc, red);
  if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// ---------------------------------------------------------------------------
// K6: tridiagonal eigen-solve (tridiag.cuh).
// Lowest eigenvalue by multisection; optional convergence test against the previous
// check, which sets the stop flag. The bracket starts from the previous check: by
// interlacing the lowest Ritz value only moves down as the tridiagonal grows, so one
// point just above it and 31 at geometric distances below it (2^-52 .. 2^8 of the
// spectrum's scale) bracket it in one round. The first check, or a probe that fails to
// bracket, starts from the Gershgorin interval.
__global__ void __launch_bounds__(TRI_THREADS) k_tri_lowest(Scal S, int check_conv, double tol, int slot, int level) {
  __shared__ double br[2];
  const int m = S.flags[2];
  if (m <= 0) return;
  const int lane = threadIdx.x & 31;
  const Tri T = tri_stage(S.alpha, S.beta, m, level);
  double lo = T.glo, hi = T.ghi;
  const double prev = slot > 0 ? S.ritz[slot - 1] : 0.0;
  if (slot > 0 && prev >= T.glo && prev <= T.ghi) {
    if (threadIdx.x < 32) {
      const double scale = fmax(T.ghi - T.glo, fabs(prev));
      // lane 0 just above prev (an eigenvalue lies below it), lanes 1..31 below
      const double x = lane == 0 ? prev + scale * 0x1p-48 : prev - scale * ldexp(1.0, 2 * (lane - 1) - 52);
      const unsigned hit = __ballot_sync(0xffffffffu, tri_count(T, x) >= 1);
      // counts grow with x, i.e. towards lane 0: the lanes with a hit are 0 .. L-1
      const int L = __popc(hit);
      const double xa = __shfl_sync(0xffffffffu, x, L > 0 ? L - 1 : 0);
      const double xb = __shfl_sync(0xffffffffu, x, L < 32 ? L : 31);
      if (L > 0 && L < 32 && hit == ((1u << L) - 1u)) {
        hi = xa;
        lo = xb;
      }
      if (lane == 0) {
        br[0] = lo;
        br[1] = hi;
      }
    }
    __syncthreads();
    lo = br[0];
    hi = br[1];
  }
  tri_multisect(T, lo, hi, 16);
  if (threadIdx.x == 0) {
    const double e = 0.5 * (lo + hi);
    S.ritz[slot] = e;
    S.flags[5] = m;  // the tridiagonal size this value belongs to
    if (check_conv && slot > 0 && !S.flags[0]) {
      if (fabs(e - prev) <= tol) S.flags[0] = 1;
    }
  }
}

// Lowest eigenvalue of the m x m tridiagonal: 32-point multisection from the
// Gershgorin interval to 2 ulp: *out. When the last convergence check (ritz[last],
// recorded for size flags[5]) already found it for this m, that value is taken instead
// (the same 2-ulp multisection). 200 x 200: 1147 -> 442 us.
__global__ void __launch_bounds__(TRI_THREADS) k_tri_min(const double* a, const double* b, int m, double* out,
                                                         int level, const double* ritz, const int* flags, int last) {
  if (last >= 0 && flags[5] == m) {
    if (threadIdx.x == 0) *out = ritz[last];
    return;
  }
  const Tri T = tri_stage(a, b, m, level);
  double lo = T.glo, hi = T.ghi;
  tri_multisect(T, lo, hi, 24);
  if (threadIdx.x == 0) *out = 0.5 * (lo + hi);
}

// All eigenvalues (ascending), a warp for each: 32-point multisection until the
// interval's ends are neighbours, 12 rounds where one thread's bisection took 53, and
// the FP64 pipes of all SMs (200 x 200 with the vector: 10.3 -> 1.6 ms).
__global__ void __launch_bounds__(32) k_tri_all(const double* a, const double* b, int m, double* eig, int level) {
  const Tri T = tri_stage(a, b, m, level);
  const int lane = threadIdx.x, k = blockIdx.x;
  double lo = T.glo, hi = T.ghi;
  for (int it = 0; it < 200; it++) {
    const double x = lo + (hi - lo) * (lane + 1) / 33.0;
    const unsigned hit = __ballot_sync(0xffffffffu, tri_count(T, x) > k);
    const int f = hit ? __ffs(hit) - 1 : 32;
    const double xf = __shfl_sync(0xffffffffu, x, f < 32 ? f : 31);
    const double xp = __shfl_sync(0xffffffffu, x, f > 0 ? f - 1 : 0);
    const double nhi = f < 32 ? xf : hi, nlo = f > 0 ? xp : lo;
    if (nhi == hi && nlo == lo) break;
    hi = nhi;
    lo = nlo;
  }
  if (lane == 0) eig[k] = 0.5 * (lo + hi);
}

// Eigenvector for eigenvalue *lam_p by inverse iteration. With `staged` everything
// lives in shared memory (8 m doubles) and only the result is written out (200 x 200:
// 877 -> 469 us); else one thread works in global memory.
__global__ void __launch_bounds__(32) k_tri_vec(const double* a, const double* b, int m, const double* lam_p,
                                                double* y, double* work, int staged) {
  if (!staged) {
    if (threadIdx.x == 0) tri_inverse_iteration(a, b, m, *lam_p, y, work);
    return;
  }
  extern __shared__ double tri_sm[];
  tri_inverse_warp(a, b, m, *lam_p, tri_sm);
  for (int i = threadIdx.x; i < m; i += 32) y[i] = tri_sm[2 * m + i];
}

// psi[r] = sum_l y[l] V_l[r] (GEMV over the Krylov basis); partial |psi|^2.
template <bool CPLX>
__global__ void k_ritz(const double* __restrict__ V, int64_t dim, int m, const double* __restrict__ y,
                       double* __restrict__ psi, double* __restrict__ part_norm) {
  extern __shared__ double ys[];
  for (int t = threadIdx.x; t < m; t += blockDim.x) ys[t] = y[t];
  __syncthreads();
  double nn = 0;
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < dim) {
    if (CPLX) {
      double2 acc = make_double2(0, 0);
      for (int k = 0; k < m; k++) {
        const double2 v = reinterpret_cast<const double2*>(V)[(int64_t)k * dim + r];
        acc.x += ys[k] * v.x;
        acc.y += ys[k] * v.y;
      }
      reinterpret_cast<double2*>(psi)[r] = acc;
      nn = acc.x * acc.x + acc.y * acc.y;
    } else {
      double acc = 0;
      for (int k = 0; k < m; k++) acc += ys[k] * V[(int64_t)k * dim + r];
      psi[r] = acc;
      nn = acc * acc;
    }
  }
  __shared__ double red[8];
  for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = nn;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int i = 0; i < (int)(blockDim.x / 32); i++) s += red[i];
    part_norm[blockIdx.x] = s;
  }
}

// Device start vector: u - 1/2 with u uniform in (0, 1) from splitmix64 of
// (seed, index) (Steele, Lea, Flood 2014), so the start costs no host work.
__global__ void k_rand_fill(double* x, int64_t n, uint64_t seed) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t z = seed * 0x9E3779B97F4A7C15ULL + (uint64_t)(i + 1) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    x[i] = ((double)(z >> 11) + 0.5) * (1.0 / 9007199254740992.0) - 0.5;
  }
}

// out = conj(psi) (interleaved complex; a copy when real).
__global__ void k_conj(const double* __restrict__ psi, double* __restrict__ out, int64_t n, int cplx) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (cplx && (i & 1)) ? -psi[i] : psi[i];
}

__global__ void k_sum(const double* part, int n, double* out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0;
    for (int i = 0; i < n; i++) s += part[i];
    *out = s;
  }
}

__global__ void k_scale_by_norm(double* v, int64_t n, const double* nrm2) {
  const double inv = 1.0 / sqrt(*nrm2);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v[i] *= inv;
}

// partial Re<a, b> over blocks (real or interleaved complex, n doubles)
__global__ void k_dot_partial(const double* a, const double* b, int64_t n, int cplx, double* part) {
  double s = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    s += a[i] * b[i];  // Re(conj(a) b) = ar br + ai bi for interleaved complex
  (void)cplx;
  __shared__ double red[8];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0;
    for (int i = 0; i < (int)(blockDim.x / 32); i++) t += red[i];
    part[blockIdx.x] = t;
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// MT19937 (Matsumoto & Nishimura 1998) and its 64-bit variant (Nishimura 2000),
// written from the published algorithms: the streams std::mt19937 and the
// reference's genrand64_real3 produce for a given seed.
namespace {
struct MT32 {
  uint32_t s[624];
  int i = 624;
  explicit MT32(uint32_t seed) {
    s[0] = seed;
    for (int k = 1; k < 624; k++) s[k] = 1812433253u * (s[k - 1] ^ (s[k - 1] >> 30)) + (uint32_t)k;
  }
  uint32_t next() {
    if (i >= 624) {
      for (int k = 0; k < 624; k++) {
        const uint32_t y = (s[k] & 0x80000000u) | (s[(k + 1) % 624] & 0x7fffffffu);
        s[k] = s[(k + 397) % 624] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
      }
      i = 0;
    }
    uint32_t y = s[i++];
    y ^= y >> 11;
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    y ^= y >> 18;
    return y;
  }
};
struct MT64 {
  uint64_t s[312];
  int i = 312;
  explicit MT64(uint64_t seed) {
    s[0] = seed;
    for (int k = 1; k < 312; k++) s[k] = 6364136223846793005ULL * (s[k - 1] ^ (s[k - 1] >> 62)) + (uint64_t)k;
  }
  uint64_t next() {
    if (i >= 312) {
      for (int k = 0; k < 312; k++) {
        const uint64_t y = (s[k] & 0xFFFFFFFF80000000ULL) | (s[(k + 1) % 312] & 0x7FFFFFFFULL);
        s[k] = s[(k + 156) % 312] ^ (y >> 1) ^ ((y & 1ULL) ? 0xB5026F5AA96619E9ULL : 0ULL);
      }
      i = 0;
    }
    uint64_t x = s[i++];
    x ^= (x >> 29) & 0x5555555555555555ULL;
    x ^= (x << 17) & 0x71D67FFFEDA60000ULL;
    x ^= (x << 37) & 0xFFF7EEE000000000ULL;
    x ^= x >> 43;
    return x;
  }
  double real3() { return ((double)(next() >> 12) + 0.5) * (1.0 / 4503599627370496.0); }
};

// The reference writes phi_0[i] = complex<double>(draw() - 0.5, draw() - 0.5)
// (lanczos_hamiltonian.cpp:468-476, matrix.cpp:54-70); GCC, which builds it,
// evaluates the two arguments right to left, so the imaginary part is drawn
// first (its recorded Lanczos coefficients in complex sectors agree with this
// order only). Complex sectors follow that order; real sectors, which the
// library runs in real arithmetic, take one draw per entry.
void fill_start(uint64_t seed, int rng, int64_t dim, int cplx, double* out) {
  const int64_t n = dim * (cplx ? 2 : 1);
  double nrm = 0;
  MT32 g32((uint32_t)seed);
  MT64 g64(rng == 0 ? 0 : seed);
  auto draw = [&]() { return rng == 0 ? g32.next() * 1.0 / 4294967295.0 - 0.5 : g64.real3() - 0.5; };
  for (int64_t i = 0; i < n; i += (cplx ? 2 : 1)) {
    if (cplx) {
      out[i + 1] = draw();
      out[i] = draw();
      nrm += out[i] * out[i] + out[i + 1] * out[i + 1];
    } else {
      out[i] = draw();
      nrm += out[i] * out[i];
    }
  }
  nrm = sqrt(nrm);
  for (int64_t i = 0; i < n; i++) out[i] /= nrm;
}
}  // namespace

// ---------------------------------------------------------------------------
struct blqh_lanczos {
  blqh_ctx* ctx = nullptr;
  const blqh_csr* M = nullptr;
  blqh_lanczos_opts o{};
  int64_t dim = 0;
  int cplx = 0, vw = 1;
  int mmax = 0;
  double* V = nullptr;     // [(mmax+1) * dim * vw]
  double* w = nullptr;     // [dim * vw]
  double* psi = nullptr;   // [dim * vw]
  double* scal = nullptr;  // scalar block
  Scal S{};
  double* part = nullptr;  // dot partials [nblk_dot * (mmax+1) * 2]
  double* pnorm = nullptr; // [max(nblk_dot, nblk_upd)]
  double2* apart = nullptr;  // partials of h_j (at most 2 blocks per SM)
  double* npart = nullptr;   // [ntile] partials of |w|^2 after the three-term step
  double* work = nullptr;  // tridiagonal work [5*mmax + ...]
  double* y = nullptr;     // [mmax] Ritz coefficients
  float2* xs = nullptr;    // [dim * vw] (hi, lo) split of the SpMV input (double-float accumulation)
  FixedMatrix fx;          // the matrix in fixed point (complex FP64 matrices)
  int2* xq = nullptr;      // [dim * 2] the SpMV input in fixed point, then xe and pmax in the same buffer
  int* xe = nullptr;       // the exponent that its entries are below
  unsigned* pmax = nullptr;  // [nblk_upd] block maxima of |w| (high words), where its scale comes from
  // complex sectors: fixed-point planes of V and, in the last row, of w (or null)
  int* Q1 = nullptr;       // [(mmax+2) * pld]
  int* Q0 = nullptr;
  int* QE = nullptr;       // [(mmax+2) * ntile] tile exponents
  int tile = 0, ntile = 0; // doubles per tile, tiles of a vector
  int64_t pld = 0;         // plane row stride: ntile * tile
  // real sectors: FP32 planes of V for the Gram-Schmidt pass, hi and (double-float dots) lo (or null)
  float* Vh = nullptr;     // [(mmax+1) * vld]
  float* Vl = nullptr;
  int64_t vld = 0;         // plane row stride (floats): dim rounded up to a multiple of 4
  int nblk_dot = 0, nblk_upd = 0;  // 1024-row tiles; blocks of the ordered update
  int steps = 0;
  int last_check = -1;  // ritz[] slot of the last convergence check of the last run (-1: none)
  bool started = false, iterated = false, have_psi = false;
};

namespace {

void free_lanczos(blqh_lanczos* L) {
  if (!L) return;
  dev_free(L->xs);
  fixed_release(&L->fx);
  dev_free(L->xq);
  dev_free(L->Q1);
  dev_free(L->Q0);
  dev_free(L->QE);
  dev_free(L->Vh);
  dev_free(L->Vl);
  dev_free(L->V);
  dev_free(L->w);
  dev_free(L->psi);
  dev_free(L->scal);
  dev_free(L->part);
  dev_free(L->pnorm);
  dev_free(L->apart);
  dev_free(L->npart);
  dev_free(L->work);
  dev_free(L->y);
  delete L;
}

int spmv_lpr(double mean_row) {
  if (mean_row >= 96) return 32;
  if (mean_row >= 40) return 16;
  if (mean_row >= 16) return 8;
  return 4;
}

template <class VT, bool CPLX>
void spmv_t(blqh_ctx* ctx, const blqh_csr* M, const double* x, double* y, const double* bptr, const double* xprev,
            const int* stop) {
  const int lpr = M->lanes_per_row;
  const int threads = 256;
  const int64_t groups = M->dim;
  int64_t blocks = (groups * lpr + threads - 1) / threads;
  const int64_t cap = (int64_t)ctx->num_sms * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  auto rp = M->d_row_ptr;
  auto cl = M->d_col;
  auto vl = reinterpret_cast<const VT*>(M->d_val);
  switch (lpr) {
    case 32: k_spmv<VT, CPLX, 32><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, x, y, M->dim, bptr, xprev, stop); break;
    case 16: k_spmv<VT, CPLX, 16><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, x, y, M->dim, bptr, xprev, stop); break;
    case 8: k_spmv<VT, CPLX, 8><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, x, y, M->dim, bptr, xprev, stop); break;
    default: k_spmv<VT, CPLX, 4><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, x, y, M->dim, bptr, xprev, stop); break;
  }
}

template <bool CPLX>
void spmv_df_t(blqh_ctx* ctx, const blqh_csr* M, const float2* xs, double* y, const double* bptr,
               const double* xprev, const int* stop) {
  if (M->blk_state > 0 && blocked_mode() >= 0) {
    blocked_spmv(ctx, M, xs, y, bptr, xprev, stop);
    return;
  }
  const int lpr = M->lanes_per_row;
  const int threads = 256;
  int64_t blocks = (M->dim * lpr + threads - 1) / threads;
  const int64_t cap = (int64_t)ctx->num_sms * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  auto rp = M->d_row_ptr;
  auto cl = M->d_col;
  auto vl = reinterpret_cast<const float*>(M->d_val);
  if (!CPLX && lpr >= 8) {
    if (lpr == 32)
      k_spmv_df_v4<32><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, xs, y, M->dim, bptr, xprev, stop);
    else if (lpr == 16)
      k_spmv_df_v4<16><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, xs, y, M->dim, bptr, xprev, stop);
    else
      k_spmv_df_v4<8><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, xs, y, M->dim, bptr, xprev, stop);
    return;
  }
  switch (lpr) {
    case 32: k_spmv_df<CPLX, 32><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, xs, y, M->dim, bptr, xprev, stop); break;
    case 16: k_spmv_df<CPLX, 16><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, xs, y, M->dim, bptr, xprev, stop); break;
    case 8: k_spmv_df<CPLX, 8><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, xs, y, M->dim, bptr, xprev, stop); break;
    default: k_spmv_df<CPLX, 4><<<(int)blocks, threads, 0, ctx->stream>>>(rp, cl, vl, xs, y, M->dim, bptr, xprev, stop); break;
  }
}

// y = H x - b xprev. With an FP32-valued CSR and a split buffer xs, the product
// accumulates in double-float (k_spmv_df); with a fixed-point copy fx of the matrix and
// buffers xq, xe, pmax (|x| <= 1) in integers (k_spmv_fixed); otherwise in native FP64 (k_spmv).
void spmv_dev(blqh_ctx* ctx, const blqh_csr* M, const double* x, double* y, const double* bptr = nullptr,
              const double* xprev = nullptr, const int* stop = nullptr, float2* xs = nullptr,
              bool xs_ready = false, const FixedMatrix* fx = nullptr, int2* xq = nullptr, int* xe = nullptr,
              unsigned* pmax = nullptr) {
  if (xs && M->precision == BLQH_VAL_FP32) {
    const int64_t n = M->dim * (M->is_complex ? 2 : 1);
    if (!xs_ready) {  // else the caller's previous kernel left x's split in xs
      TimerScope tm(ctx, TM_MISC);
      k_split<<<grid_for(ctx, n, 256, 8), 256, 0, ctx->stream>>>(x, xs, n, stop);
      count_launch(ctx, TM_MISC);
    }
    TimerScope ts(ctx, TM_SPMV);
    if (M->is_complex) spmv_df_t<true>(ctx, M, xs, y, bptr, xprev, stop);
    else spmv_df_t<false>(ctx, M, xs, y, bptr, xprev, stop);
    BLQH_TRY_CUDA(ctx, cudaGetLastError());
    count_launch(ctx, TM_SPMV);
    return;
  }
  if (xq) {  // fixed point (complex FP64)
    if (!xs_ready) fixed_vector(ctx, x, xq, xe, pmax, M->dim * 2, stop);
    TimerScope ts(ctx, TM_SPMV);
    fixed_spmv(ctx, M, *fx, x, xq, xe, y, bptr, xprev, stop);
    BLQH_TRY_CUDA(ctx, cudaGetLastError());
    count_launch(ctx, TM_SPMV);
    return;
  }
  TimerScope ts(ctx, TM_SPMV);
  if (M->is_complex) {
    if (M->precision == BLQH_VAL_FP64) spmv_t<double2, true>(ctx, M, x, y, bptr, xprev, stop);
    else spmv_t<float2, true>(ctx, M, x, y, bptr, xprev, stop);
  } else {
    if (M->precision == BLQH_VAL_FP64) spmv_t<double, false>(ctx, M, x, y, bptr, xprev, stop);
    else spmv_t<float, false>(ctx, M, x, y, bptr, xprev, stop);
  }
  BLQH_TRY_CUDA(ctx, cudaGetLastError());
  count_launch(ctx, TM_SPMV);
}

// Dynamic shared memory of the tridiagonal kernels: `per` doubles per Lanczos
// step when that and the kernel's `fixed` bytes of static shared memory fit in
// 48 KB, else 0 (they then read global memory).
int tri_smem(const blqh_lanczos* L, int per, size_t fixed = 0) {
  const size_t b = (size_t)per * (L->mmax + 1) * sizeof(double);
  return b + fixed <= 48 * 1024 ? (int)b : 0;
}

// What tri_stage has room for next to k_tri_lowest's bracket.
int tri_level(const blqh_lanczos* L) {
  const size_t bracket = 2 * sizeof(double);
  return tri_smem(L, 4, bracket) > 0 ? 4 : tri_smem(L, 2, bracket) > 0 ? 2 : 0;
}

// A kernel of the step chain: its blocks may be placed while the previous kernel
// on the stream drains; it waits for that kernel's results itself (pdl_begin).
template <class... P, class... A>
void launch_chained(blqh_ctx* ctx, void (*kern)(P...), int grid, int block, size_t smem, A... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  BLQH_TRY_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
}

// Rows of the planes: vector k, and w after the stored vectors.
int* q1_row(const blqh_lanczos* L, int k) { return L->Q1 ? L->Q1 + (int64_t)k * L->pld : nullptr; }
int* q0_row(const blqh_lanczos* L, int k) { return L->Q0 ? L->Q0 + (int64_t)k * L->pld : nullptr; }
int* qe_row(const blqh_lanczos* L, int k) { return L->QE ? L->QE + (int64_t)k * L->ntile : nullptr; }

NextVec next_vec(const blqh_lanczos* L, int k) {
  return {L->V + (int64_t)k * L->dim * L->vw, L->M->precision == BLQH_VAL_FP32 ? L->xs : nullptr, L->xq,
          L->xe, q1_row(L, k), q0_row(L, k), qe_row(L, k)};
}

// The step after the SpMV on the fixed-point planes (complex sectors).
template <int TILE>
void gs_step_q(blqh_lanczos* L, int j) {
  blqh_ctx* ctx = L->ctx;
  constexpr bool LOCAL = TILE == 256;
  const int64_t n = L->dim * 2;
  const double* vj = L->V + (int64_t)j * n;
  const int nk = j + 1, wr = L->mmax + 1, ng = (nk + DOT_GROUP - 1) / DOT_GROUP;
  const int na = grid_for(ctx, L->dim, 1024, 2);
  const WTile W{vj, L->w, L->apart, na, q1_row(L, wr), q0_row(L, wr), qe_row(L, wr), L->npart};
  launch_chained(ctx, k_alpha, na, 256, 0, vj, L->w, L->dim, L->apart, L->S);
  if constexpr (!LOCAL)
    launch_chained(ctx, k_local<TILE>, L->ntile, TILE / 4, 0, vj, L->w, n, L->apart, na, q1_row(L, wr),
                   q0_row(L, wr), qe_row(L, wr), L->npart, L->S, j);
  launch_chained(ctx, k_dots_q<TILE, LOCAL>, ng * L->ntile, 256, 0, L->Q1, L->Q0, L->QE, L->pld, L->ntile, n,
                 nk, ng, W, L->part, L->S, j);
  const size_t hsm = (size_t)nk * 2 * sizeof(float);
  auto update = [&](auto kern, int threads) {
    launch_chained(ctx, kern, L->ntile, threads, hsm, L->V, L->Q1, L->QE, L->pld, L->ntile, n, nk, W, L->w, L->pnorm,
                   L->S, j, 1e-13, next_vec(L, j + 1));
  };
  // One slice of vectors per block once the tiles alone give every SM two blocks, else four slices.
  // us per step, product included, one against four, runs of 100 and 250 steps: 100,141 rows (196 tiles)
  // 170 : 168 and 213 : 203; 143,143 rows (280) 200 : 197 and 252 : 244; 204,660 rows (400) 305 : 309 and
  // 373 : 375; 322,203 rows (630) 451 : 474 and 553 : 577.
  if constexpr (LOCAL) update(k_update_q<256, 16, true>, 1024);
  else if (L->ntile >= 2 * ctx->num_sms) update(k_update_q<1024, 1, false>, 256);
  else update(k_update_q<1024, 4, false>, 1024);
  count_launch(ctx, TM_REORTH, LOCAL ? 3 : 4);
}

NextPlanes next_planes(const blqh_lanczos* L, int k) {
  return {L->V + (int64_t)k * L->dim * L->vw, L->M->precision == BLQH_VAL_FP32 ? L->xs : nullptr, L->xq,
          L->xe, L->Vh ? L->Vh + (int64_t)k * L->vld : nullptr, L->Vl ? L->Vl + (int64_t)k * L->vld : nullptr, L->vld};
}

// The step after the SpMV in the fixed order of operations (real sectors, and
// complex ones without fixed-point planes).
template <bool CPLX>
void gs_step_o(blqh_lanczos* L, int j) {
  blqh_ctx* ctx = L->ctx;
  const int64_t n = L->dim * L->vw;
  const double* vj = L->V + (int64_t)j * n;
  const int nt = L->nblk_dot, nu = L->nblk_upd;
  const bool df = L->Vl != nullptr;  // double-float dots, four entries per thread in the updates
  double* apart = reinterpret_cast<double*>(L->apart);
  launch_chained(ctx, k_alpha_o<CPLX>, nt, 32, 0, vj, L->w, L->dim, apart, L->S);
  const int lg = std::min(nu, 4 * ctx->num_sms);
  if (df)
    launch_chained(ctx, k_local_o<false, 4>, lg, 256, 0, vj, L->w, L->dim, apart, nt, L->pnorm, L->pmax, nu, L->S,
                   j);
  else
    launch_chained(ctx, k_local_o<CPLX, 1>, lg, 256, 0, vj, L->w, L->dim, apart, nt, L->pnorm, L->pmax, nu, L->S,
                   j);
  if (L->o.reorth) {
    const int nk = j + 1;
    // few tiles: 8 vectors per block (one per warp), summed by each group's last block; beyond, a
    // kernel for the sums, and more vectors per block once the blocks would fill the GPU over and over:
    // 4 times for double-float dots (staging w's tile splits it), 16 for FP64 ones (32 at least: 4 per warp).
    // us per step, product included, last block against kernel, runs of 100 and 200 steps. Real FP64 dots:
    // 98 tiles 144 : 173 and 154 : 180; 315 tiles 340 : 352 and 380 : 384; 632 tiles 1024 : 1028 and
    // 1104 : 1098; 1,062 tiles 925 : 923 and 1059 : 1050. Double-float: 35 tiles 50.5 : 51.3 and 59.1 : 58.7;
    // 59 tiles 92.8 : 92.6 and 102 : 101; 140 tiles 151 : 147 and 167 : 163 (the complex FP64 pass, taken
    // where there is no room for planes, keeps that line).
    const int finish = nt <= (df || CPLX ? 64 : 512);
    const int step = finish || df || CPLX ? 8 : 32;
    const int waves = (int)((int64_t)nt * ((nk + step - 1) / step) / ((df ? 4 : 16) * ctx->num_sms));
    const int gk = step * (finish ? 1 : std::max(1, waves)), ng = (nk + gk - 1) / gk;
    auto dots = [&](auto kern) {
      launch_chained(ctx, kern, ng * nt, 256, 0, L->V, L->Vh, L->Vl, L->vld, L->dim, nt, nk, gk, ng, L->w, L->part,
                     L->pnorm, nu, finish, L->S, j);
      if (!finish) launch_chained(ctx, k_reduce_o<CPLX>, nk, 256, 0, L->part, nt, L->pnorm, nu, L->S, j);
    };
    const size_t hsm = 2 * nk * (sizeof(double) + sizeof(float));
    auto update = [&](auto kern) {
      launch_chained(ctx, kern, nu, 256, hsm, L->V, L->Vh, L->vld, L->dim, nk, L->w, L->pnorm, L->pmax, L->S);
    };
    if constexpr (CPLX) {
      dots(k_dots_o<true, false, 1>);
      update(k_update_o<true, 1, false>);
    } else if (df) {
      dots(k_dots_o<false, true, 1>);
      update(k_update_o<false, 4, true>);
    } else {
      if (finish) dots(k_dots_o<false, false, 1>);
      else dots(k_dots_o<false, false, 4>);
      if (L->Vh) update(k_update_o<false, 1, true>);
      else update(k_update_o<false, 1, false>);
    }
    count_launch(ctx, TM_REORTH, finish ? 2 : 3);
  }
  launch_chained(ctx, k_scale_o, grid_for(ctx, n, 256, 2), 256, 0, L->w, n, 0, L->pnorm, L->pmax, nu, L->S, j, 1e-13,
                 next_planes(L, j + 1));
  count_launch(ctx, TM_REORTH, 3);
}

void lanczos_step(blqh_lanczos* L, int j) {
  blqh_ctx* ctx = L->ctx;
  const int64_t n = L->dim * L->vw;
  double* vj = L->V + (int64_t)j * n;
  const double* vprev = j > 0 ? L->V + (int64_t)(j - 1) * n : nullptr;
  // from the second step on, the previous step left v_j's split in xs
  spmv_dev(ctx, L->M, vj, L->w, j > 0 ? L->S.beta + j : nullptr, vprev, L->S.flags, L->xs, j > 0,
           &L->fx, L->xq, L->xe, L->pmax);
  // three-term step: the SpMV removed beta_j v_{j-1}; remove the v_j component
  // (alpha_j). With reorth, one classical Gram-Schmidt pass against every stored
  // vector follows; taking the local step first keeps that pass from having to
  // be repeated (the norm drop of the alpha_j removal no longer enters it). The
  // step's last norm also sets beta_{j+1} (breakdown below 1e-13 of |alpha_j| + beta_j).
  TimerScope ts(ctx, TM_REORTH);
  if (L->Q1) L->tile == 1024 ? gs_step_q<1024>(L, j) : gs_step_q<256>(L, j);
  else L->cplx ? gs_step_o<true>(L, j) : gs_step_o<false>(L, j);
}

void iterate_impl(blqh_lanczos* L) {
  blqh_ctx* ctx = L->ctx;
  cudaStream_t st = ctx->stream;
  if (!L->started) {
    const int64_t n = L->dim * L->vw;
    if (L->o.rng == 2) {
      TimerScope tm(ctx, TM_MISC);
      const int blocks = grid_for(ctx, n, 256, 4);
      k_rand_fill<<<grid_for(ctx, n, 256, 8), 256, 0, st>>>(L->V, n, L->o.seed);
      k_dot_partial<<<blocks, 256, 0, st>>>(L->V, L->V, n, 0, L->pnorm);
      k_sum<<<1, 1, 0, st>>>(L->pnorm, blocks, L->S.nrm + 2);
      k_scale_by_norm<<<grid_for(ctx, n, 256, 8), 256, 0, st>>>(L->V, n, L->S.nrm + 2);
      BLQH_TRY_CUDA(ctx, cudaGetLastError());
      count_launch(ctx, TM_MISC, 4);
    } else {
      std::vector<double> x(n);
      fill_start(L->o.seed, L->o.rng, L->dim, L->cplx, x.data());
      BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(L->V, x.data(), x.size() * 8, cudaMemcpyHostToDevice, st));
      BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(st));
    }
    L->started = true;
  }
  BLQH_TRY_CUDA(ctx, cudaMemsetAsync(L->S.flags, 0, 4 * sizeof(int), st));
  BLQH_TRY_CUDA(ctx, cudaMemsetAsync(L->S.flags + 5, 0xFF, sizeof(int), st));  // no check's size yet
  if (L->Q1 || L->Vh) {  // planes of the start vector (the steps write the others)
    TimerScope tm(ctx, TM_MISC);
    const int64_t n = L->dim * L->vw;
    if (L->Q1)
      launch_chained(ctx, L->tile == 1024 ? k_planes_q<1024> : k_planes_q<256>, L->ntile, L->tile / 4, 0, L->V, n,
                     next_vec(L, 0));
    else
      launch_chained(ctx, k_scale_o, grid_for(ctx, n, 256, 2), 256, 0, L->V, n, 1, nullptr, nullptr, 0, L->S, 0,
                     0.0, next_planes(L, 0));
    count_launch(ctx, TM_MISC);
  }
  BLQH_TRY_CUDA(ctx, cudaMemsetAsync(L->S.beta, 0, sizeof(double), st));
  const int chunk = std::max(1, L->o.check_every);
  const bool conv = L->o.tol > 0;
  int* hflags = reinterpret_cast<int*>(ctx->pinned);
  cudaEvent_t ev[2];
  cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming);
  cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming);
  int launched_chunks = 0;
  int j = 0;
  bool stop = false;
  while (j < L->mmax && !stop) {
    const int jend = std::min(L->mmax, j + chunk);
    for (; j < jend; j++) lanczos_step(L, j);
    if (conv) {  // with tol = 0 the recurrence runs to max_steps: no check needed
      TimerScope tm(ctx, TM_MISC);
      k_tri_lowest<<<1, TRI_THREADS, tri_smem(L, tri_level(L)), st>>>(L->S, 1, L->o.tol, launched_chunks, tri_level(L));
      BLQH_TRY_CUDA(ctx, cudaGetLastError());
      count_launch(ctx, TM_MISC);
    }
    int* slot = hflags + 4 * (launched_chunks & 1);
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(slot, L->S.flags, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
    BLQH_TRY_CUDA(ctx, cudaEventRecord(ev[launched_chunks & 1], st));
    launched_chunks++;
    // wait for the previous chunk's flags (the current chunk keeps the GPU busy)
    if (launched_chunks >= 2) {
      const int prev = (launched_chunks - 2) & 1;
      BLQH_TRY_CUDA(ctx, cudaEventSynchronize(ev[prev]));
      if (hflags[4 * prev]) stop = true;
    }
  }
  BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(st));
  cudaEventDestroy(ev[0]);
  cudaEventDestroy(ev[1]);
  int f[4];
  BLQH_TRY_CUDA(ctx, cudaMemcpy(f, L->S.flags, sizeof(f), cudaMemcpyDeviceToHost));
  L->steps = f[2];
  L->last_check = conv && launched_chunks > 0 ? launched_chunks - 1 : -1;
  L->iterated = true;
  L->have_psi = false;
}

void ritz_impl(blqh_lanczos* L) {
  blqh_ctx* ctx = L->ctx;
  cudaStream_t st = ctx->stream;
  const int m = L->steps;
  TimerScope tm(ctx, TM_MISC);
  // only the lowest Ritz pair is needed here (blqh_lanczos_eig gives them all)
  const int lv = tri_level(L);
  k_tri_min<<<1, TRI_THREADS, tri_smem(L, lv), st>>>(L->S.alpha, L->S.beta, m, L->work + 6 * L->mmax, lv, L->S.ritz,
                                                     L->S.flags, L->last_check);
  k_tri_vec<<<1, 32, tri_smem(L, 8), st>>>(L->S.alpha, L->S.beta, m, L->work + 6 * L->mmax, L->y, L->work,
                                            tri_smem(L, 8) > 0);
  const int blocks = (int)((L->dim + 255) / 256);
  if (L->cplx)
    k_ritz<true><<<blocks, 256, m * sizeof(double), st>>>(L->V, L->dim, m, L->y, L->psi, L->pnorm);
  else
    k_ritz<false><<<blocks, 256, m * sizeof(double), st>>>(L->V, L->dim, m, L->y, L->psi, L->pnorm);
  k_sum<<<1, 1, 0, st>>>(L->pnorm, blocks, L->S.nrm + 2);
  k_scale_by_norm<<<grid_for(ctx, L->dim * L->vw, 256, 8), 256, 0, st>>>(L->psi, L->dim * L->vw, L->S.nrm + 2);
  BLQH_TRY_CUDA(ctx, cudaGetLastError());
  count_launch(ctx, TM_MISC, 5);
  L->have_psi = true;
}

// <x|H|x> with the stored CSR values (x normalized, on the device).
double rq_stored(blqh_lanczos* L, const double* x) {
  blqh_ctx* ctx = L->ctx;
  cudaStream_t st = ctx->stream;
  spmv_dev(ctx, L->M, x, L->w);
  const int64_t n = L->dim * L->vw;
  const int blocks = grid_for(ctx, n, 256, 4);
  TimerScope tm(ctx, TM_MISC);
  k_dot_partial<<<blocks, 256, 0, st>>>(x, L->w, n, L->cplx, L->pnorm);
  k_sum<<<1, 1, 0, st>>>(L->pnorm, blocks, L->S.nrm + 3);
  count_launch(ctx, TM_MISC, 2);
  double e = 0;
  BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(&e, L->S.nrm + 3, 8, cudaMemcpyDeviceToHost, st));
  BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(st));
  return e;
}

// K10 for the SpMV of a matrix of at least 2^15 rows: the row kernel at 4, 8,
// 16 and 32 lanes per row and, for FP32 values with double-float accumulation,
// the blocked kernel (spmv_blocked.cu) are timed on this matrix (x = 0, three
// products each); the choice is cached per class as (lanes, blocked).
// BLQH_SPMV_BLOCKED=1 forces the blocked kernel, =0 rules it out.
void tune_spmv(blqh_lanczos* L) {
  blqh_csr* M = const_cast<blqh_csr*>(L->M);
  blqh_ctx* ctx = L->ctx;
  const int bm = blocked_mode();
  const bool can_blk = M->precision == BLQH_VAL_FP32 && L->xs && bm >= 0;
  if (can_blk && bm == 1) {
    blocked_prepare(ctx, M);
    return;
  }
  if (L->xq) return;  // fixed point: no shape to choose
  if (M->dim < (1 << 15) || !tune_enabled()) {
    if (can_blk && M->dim >= (1 << 15)) blocked_prepare(ctx, M);
    return;
  }
  const int mode = M->precision == BLQH_VAL_FP32 ? (L->o.accumulate ? 1 : 2) : 0;
  const std::string key = tune_key("spmv", mode, M->is_complex, M->dim, M->mean_row, 1);
  int lpr = 0, blk = 0;
  if (!tune_lookup(key, &lpr, &blk)) {
    const int64_t n = L->dim * L->vw;
    BLQH_TRY_CUDA(ctx, cudaMemsetAsync(L->V, 0, n * 8, ctx->stream));
    cudaEvent_t e0, e1;
    BLQH_TRY_CUDA(ctx, cudaEventCreate(&e0));
    BLQH_TRY_CUDA(ctx, cudaEventCreate(&e1));
    auto time3 = [&]() {
      spmv_dev(ctx, M, L->V, L->w, nullptr, nullptr, nullptr, L->xs);  // warm-up
      BLQH_TRY_CUDA(ctx, cudaEventRecord(e0, ctx->stream));
      for (int r = 0; r < 3; r++) spmv_dev(ctx, M, L->V, L->w, nullptr, nullptr, nullptr, L->xs);
      BLQH_TRY_CUDA(ctx, cudaEventRecord(e1, ctx->stream));
      BLQH_TRY_CUDA(ctx, cudaEventSynchronize(e1));
      float ms = 0;
      BLQH_TRY_CUDA(ctx, cudaEventElapsedTime(&ms, e0, e1));
      return (double)ms;
    };
    double best = 1e30;
    if (M->blk_state > 0) blocked_release(M);
    for (int c : {4, 8, 16, 32}) {
      M->lanes_per_row = c;
      const double ms = time3();
      if (ms < best) {
        best = ms;
        lpr = c;
      }
    }
    M->lanes_per_row = lpr;
    if (can_blk && blocked_prepare(ctx, M)) {
      const double ms = time3();
      if (blocked_error(ctx, M) == BLQH_OK && ms < best) {
        best = ms;
        blk = 1;
      }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    tune_store(key, lpr, blk, best / 3);
  }
  M->lanes_per_row = lpr;
  if (blk && can_blk) blocked_prepare(ctx, M);
  else if (M->blk_state > 0) blocked_release(M);
}

// The full Gram-Schmidt pass works on planes next to the Krylov basis (fixed point
// in complex sectors, FP32 in real ones); BLQH_GS_FP64=1 keeps it on the FP64 vectors.
bool gs_planes_enabled() {
  const char* e = getenv("BLQH_GS_FP64");
  return !(e && e[0] == '1');
}

// BLQH_RQ_REGEN=1 finishes FP32-valued runs with the regenerated FP64 elements
// (the row generator again) instead of the stored FP32 rests.
bool regen_forced() {
  const char* e = getenv("BLQH_RQ_REGEN");
  return e && e[0] == '1';
}

// <psi|H|psi> from the FP32 values and their stored FP32 rests (k_rq_res).
double rayleigh_res_impl(blqh_lanczos* L) {
  blqh_ctx* ctx = L->ctx;
  const blqh_csr* M = L->M;
  TimerScope ts(ctx, TM_BUILD);
  spmv_dev(ctx, M, L->psi, L->w, nullptr, nullptr, nullptr, L->xs);  // y = H32 psi; xs = (hi, lo) of psi
  const int grid = grid_for(ctx, M->dim * 32, 256, 8);
  if (M->is_complex)
    k_rq_res<true><<<grid, 256, 0, ctx->stream>>>(M->d_row_ptr, M->d_col, M->d_res, L->xs, L->psi, L->w, M->dim,
                                                  L->pnorm);
  else
    k_rq_res<false><<<grid, 256, 0, ctx->stream>>>(M->d_row_ptr, M->d_col, M->d_res, L->xs, L->psi, L->w, M->dim,
                                                   L->pnorm);
  BLQH_TRY_CUDA(ctx, cudaGetLastError());
  count_launch(ctx, TM_BUILD);
  std::vector<double> h(grid);
  BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(h.data(), L->pnorm, grid * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  double e = 0;
  for (int b = 0; b < grid; b++) e += h[b];
  return e;
}

blqh_lanczos* create_impl(blqh_ctx* ctx, const blqh_csr* M, const blqh_lanczos_opts& o) {
  blqh_lanczos* L = new blqh_lanczos();
  L->ctx = ctx;
  L->M = M;
  L->o = o;
  L->dim = M->dim;
  L->cplx = M->is_complex;
  L->vw = L->cplx ? 2 : 1;
  L->mmax = (int)std::min<int64_t>(o.max_steps, M->dim);
  const_cast<blqh_csr*>(M)->lanes_per_row = spmv_lpr(M->mean_row);
  const int upd_smem = 2 * (L->mmax + 1) * (int)(sizeof(double) + sizeof(float));
  smem_attr_at_least(k_update_o<false, 1, false>, upd_smem);
  smem_attr_at_least(k_update_o<false, 1, true>, upd_smem);
  smem_attr_at_least(k_update_o<false, 4, true>, upd_smem);
  smem_attr_at_least(k_update_o<true, 1, false>, upd_smem);
  const int q_smem = 2 * (L->mmax + 1) * (int)sizeof(float);
  smem_attr_at_least(k_update_q<256, 16, true>, q_smem);
  smem_attr_at_least(k_update_q<1024, 4, false>, q_smem);
  smem_attr_at_least(k_update_q<1024, 1, false>, q_smem);
  try {
    const int64_t n = L->dim * L->vw;
    L->V = dalloc<double>(ctx, (size_t)(L->mmax + 1) * n);
    L->w = dalloc<double>(ctx, n);
    L->psi = dalloc<double>(ctx, n);
    const int m = L->mmax;
    const int max_groups = m / DOT_GROUP + 2;  // vector groups of the dots, one arrival counter each
    const size_t ns = (size_t)m + (m + 1) + 2 * (m + 1) + 4 + m + 4 + (CNT_DOTS + max_groups + 1) / 2;
    L->scal = dalloc<double>(ctx, ns);
    BLQH_TRY_CUDA(ctx, cudaMemsetAsync(L->scal, 0, ns * 8, ctx->stream));
    double* p = L->scal;
    L->S.alpha = p;
    p += m;
    L->S.beta = p;
    p += m + 1;
    L->S.h2 = p;
    p += 2 * (m + 1);
    L->S.nrm = p;
    p += 4;
    L->S.ritz = p;
    p += m;
    L->S.flags = reinterpret_cast<int*>(p);
    p += 4;
    L->S.cnt = reinterpret_cast<unsigned*>(p);
    // Short tiles spread small sectors over more blocks and save a kernel per step; they cost more
    // reductions and smaller runs of loads. us per step, product included, 256 against 1024, runs of
    // 100 and 250 steps: 5,940 rows 33.8 : 38.0 and 38.7 : 41.0; 9,402 rows 38.4 : 40.2 and 44.9 : 44.9;
    // 16,024 rows 48.1 : 46.2 and 57.9 : 52.6; 30,772 rows 85.7 : 71.7 and 103 : 82.2.
    L->tile = n <= 24576 ? 256 : 1024;
    L->ntile = (int)((n + L->tile - 1) / L->tile);
    L->pld = (int64_t)L->ntile * L->tile;
    L->nblk_dot = (int)((L->dim + GS_ROWS - 1) / GS_ROWS);
    L->nblk_upd = (int)((L->dim + 255) / 256);
    L->part = dalloc<double>(ctx, (size_t)std::max(L->nblk_dot, L->ntile) * (m + 1) * 2);
    // block partials: at most one per 256 rows, or 8 per SM
    L->pnorm = dalloc<double>(ctx, std::max<int64_t>((n + 255) / 256, (int64_t)ctx->num_sms * 8) + 1024);
    L->apart = dalloc<double2>(ctx, std::max((size_t)L->nblk_dot, (size_t)ctx->num_sms * 2));
    L->npart = dalloc<double>(ctx, L->ntile);
    L->work = dalloc<double>(ctx, 8 * (size_t)m + 16);
    L->y = dalloc<double>(ctx, m + 1);
    if (M->precision == BLQH_VAL_FP32 && o.accumulate == 0) L->xs = dalloc<float2>(ctx, n + 2);
    // a fixed-point copy and planes of FP64-valued runs come on top of what those need, FP32-valued
    // runs count on theirs
    const bool fp64 = M->precision == BLQH_VAL_FP64;
    const size_t copy = (size_t)M->nnz * 16 + (size_t)M->dim * 20 + (size_t)n * 8;
    if (!o.accumulate && optional_room(ctx, copy) && fixed_prepare(ctx, M, &L->fx)) try {
        L->xq = dalloc<int2>(ctx, n + 2 + L->nblk_upd);
        L->xe = reinterpret_cast<int*>(L->xq + n);
        L->pmax = reinterpret_cast<unsigned*>(L->xq + n + 2);
      } catch (const BlqhError& e) {  // without room for it: the FP64 product
        if (e.code != BLQH_ERR_NOMEM) throw;
        fixed_release(&L->fx);
        ctx->last_error.clear();
      }
    // (real sectors with accumulate = 1 keep the FP32 plane for the correction, not for the dots)
    const size_t planes = (size_t)(m + 2) * n * (L->cplx ? 8 : 4);
    if (o.reorth && gs_planes_enabled() && !(L->cplx && o.accumulate) && (!fp64 || optional_room(ctx, planes))) {
      // the planes take up to the Krylov basis' memory again; without room for
      // them the run works on the FP64 vectors
      try {
        if (L->cplx) {
          const size_t rows = (size_t)m + 2;
          L->Q1 = dalloc<int>(ctx, rows * L->pld);
          L->Q0 = dalloc<int>(ctx, rows * L->pld);
          L->QE = dalloc<int>(ctx, rows * L->ntile);
        } else {
          L->vld = (n + 3) & ~(int64_t)3;
          L->Vh = dalloc<float>(ctx, (size_t)(m + 1) * L->vld);
          if (M->precision == BLQH_VAL_FP32 && o.accumulate == 0) {
            L->Vl = dalloc<float>(ctx, (size_t)(m + 1) * L->vld);
            L->nblk_upd = (int)((n + 1023) / 1024);
          }
        }
      } catch (const BlqhError& e) {
        if (e.code != BLQH_ERR_NOMEM) throw;
        dev_free(L->Q1);
        dev_free(L->Q0);
        dev_free(L->Vh);
        L->Q1 = L->Q0 = L->QE = nullptr;
        L->Vh = L->Vl = nullptr;
        ctx->last_error.clear();
      }
    }
    tune_spmv(L);
  } catch (const BlqhError&) {
    free_lanczos(L);
    throw;
  }
  return L;
}

// blqh_debug_dots on device pointers; part, S as in a Lanczos object of nk steps.
template <int TILE>
void debug_dots_q(blqh_ctx* ctx, DevBufs& G, const double* V, const double* w, int64_t n, int nk, double* part, Scal S) {
  constexpr bool LOCAL = TILE == 256;
  const int ntile = (int)((n + TILE - 1) / TILE), ng = (nk + DOT_GROUP - 1) / DOT_GROUP;
  const int64_t pld = (int64_t)ntile * TILE;
  int* q1 = G.add(dalloc<int>(ctx, pld * (nk + 1)));
  int* q0 = G.add(dalloc<int>(ctx, pld * (nk + 1)));
  int* qe = G.add(dalloc<int>(ctx, (size_t)ntile * (nk + 1)));
  double2* apart = G.add(dalloc<double2>(ctx, 1));
  double* npart = G.add(dalloc<double>(ctx, ntile));
  BLQH_TRY_CUDA(ctx, cudaMemsetAsync(apart, 0, sizeof(double2), ctx->stream));
  for (int k = 0; k <= nk; k++)
    launch_chained(ctx, k_planes_q<TILE>, ntile, TILE / 4, 0, k < nk ? V + k * n : w, n,
                   NextVec{nullptr, nullptr, nullptr, nullptr, q1 + k * pld, q0 + k * pld, qe + (int64_t)k * ntile});
  const WTile W{w, w, apart, 1, q1 + nk * pld, q0 + nk * pld, qe + (int64_t)nk * ntile, npart};
  launch_chained(ctx, k_dots_q<TILE, LOCAL>, ng * ntile, 256, 0, q1, q0, qe, pld, ntile, n, nk, ng, W, part, S,
                 0);
}

void debug_dots_impl(blqh_ctx* ctx, int64_t n, int nk, const double* V, const double* w, int form, double* h) {
  DevBufs G;
  const int64_t dim = n / 2;
  const int nt = (int)((dim + GS_ROWS - 1) / GS_ROWS);
  double* dV = G.add(dalloc<double>(ctx, n * nk));
  double* dw = G.add(dalloc<double>(ctx, n));
  double* part = G.add(dalloc<double>(ctx, (size_t)(n / 256 + 1) * 2 * nk));
  const size_t ns = 4 * nk + 16;
  double* p = G.add(dalloc<double>(ctx, ns));
  BLQH_TRY_CUDA(ctx, cudaMemsetAsync(p, 0, ns * 8, ctx->stream));
  Scal S{};
  S.alpha = p;
  S.h2 = p + nk;
  S.flags = reinterpret_cast<int*>(p + 3 * nk);
  S.cnt = reinterpret_cast<unsigned*>(p + 3 * nk + 4);
  double* pnorm = p + ns - 1;
  BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(dV, V, n * nk * 8, cudaMemcpyHostToDevice, ctx->stream));
  BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(dw, w, n * 8, cudaMemcpyHostToDevice, ctx->stream));
  if (form == 0) {
    launch_chained(ctx, k_dots_o<true, false, 1>, (nk + 7) / 8 * nt, 256, 0, dV, nullptr, nullptr, 0, dim, nt, nk, 8,
                   (nk + 7) / 8, dw, part, pnorm, 1, 0, S, 0);
    launch_chained(ctx, k_reduce_o<true>, nk, 256, 0, part, nt, pnorm, 1, S, 0);
  } else if (form == 1) {
    debug_dots_q<1024>(ctx, G, dV, dw, n, nk, part, S);
  } else if (form == 2) {
    debug_dots_q<256>(ctx, G, dV, dw, n, nk, part, S);
  } else {
    debug_batch_pass(ctx, dV, dw, n, nk, S.h2, false);
  }
  BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(h, S.h2, 2 * nk * 8, cudaMemcpyDeviceToHost, ctx->stream));
  BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
}

}  // namespace

extern "C" {

int blqh_debug_batch_update(blqh_ctx* ctx, int64_t n, int nk, const double* V, double* w, const double* h) {
  if (!ctx || !V || !w || !h || n < 2 || n % 2 || n > (1 << 30) || nk < 1 || nk > BLQH_MAX_LAMBDA) return BLQH_ERR_ARG;
  try {
    DevBufs G;
    double* dV = G.add(dalloc<double>(ctx, n * nk));
    double* dw = G.add(dalloc<double>(ctx, n));
    double* dh = G.add(dalloc<double>(ctx, 2 * nk));
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(dV, V, n * nk * 8, cudaMemcpyHostToDevice, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(dw, w, n * 8, cudaMemcpyHostToDevice, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(dh, h, 2 * nk * 8, cudaMemcpyHostToDevice, ctx->stream));
    debug_batch_pass(ctx, dV, dw, n, nk, dh, true);
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(w, dw, n * 8, cudaMemcpyDeviceToHost, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_debug_dots(blqh_ctx* ctx, int64_t n, int nk, const double* V, const double* w, int form, double* h) {
  if (!ctx || !V || !w || !h || n < 2 || n % 2 || n > (1 << 30) || nk < 1 || nk > BLQH_MAX_LAMBDA || form < 0 ||
      form > 3)
    return BLQH_ERR_ARG;
  try {
    debug_dots_impl(ctx, n, nk, V, w, form, h);
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_spmv(blqh_ctx* ctx, const blqh_csr* m, const double* x, double* y) {
  if (!ctx || !m || !x || !y) return BLQH_ERR_ARG;
  double* dx = nullptr;
  double* dy = nullptr;
  float2* xs = nullptr;
  int rc = BLQH_OK;
  try {
    const int64_t n = m->dim * (m->is_complex ? 2 : 1);
    dx = dalloc<double>(ctx, n);
    dy = dalloc<double>(ctx, n);
    if (m->precision == BLQH_VAL_FP32) xs = dalloc<float2>(ctx, n + 2);
    if (xs && blocked_mode() == 1) blocked_prepare(ctx, const_cast<blqh_csr*>(m));
    const_cast<blqh_csr*>(m)->lanes_per_row = spmv_lpr(m->mean_row);
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(dx, x, n * 8, cudaMemcpyHostToDevice, ctx->stream));
    spmv_dev(ctx, m, dx, dy, nullptr, nullptr, nullptr, xs);
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(y, dy, n * 8, cudaMemcpyDeviceToHost, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    rc = blocked_error(ctx, m);
  } catch (const BlqhError& e) {
    rc = e.code;
  }
  dev_free(dx);
  dev_free(dy);
  dev_free(xs);
  return rc;
}

int blqh_lanczos_create(blqh_ctx* ctx, const blqh_csr* m, const blqh_lanczos_opts* o, blqh_lanczos** out) {
  if (!ctx || !m || !o || !out) return BLQH_ERR_ARG;
  *out = nullptr;
  if (o->max_steps < 1 || o->max_steps > BLQH_MAX_LAMBDA || o->check_every < 1 || o->rng < 0 || o->rng > 2) {
    set_error(ctx, BLQH_ERR_ARG, "blqh_lanczos_create: max_steps in [1, 4096], check_every >= 1, rng 0, 1 or 2");
    return BLQH_ERR_ARG;
  }
  try {
    *out = create_impl(ctx, m, *o);
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_set_start(blqh_lanczos* L, const double* x) {
  if (!L || !x) return BLQH_ERR_ARG;
  blqh_ctx* ctx = L->ctx;
  try {
    const int64_t n = L->dim * L->vw;
    double nrm = 0;
    for (int64_t i = 0; i < n; i++) nrm += x[i] * x[i];
    if (!(nrm > 0) || !std::isfinite(nrm)) {
      set_error(ctx, BLQH_ERR_ARG, "blqh_lanczos_set_start: start vector is zero or not finite");
      return BLQH_ERR_ARG;
    }
    std::vector<double> h(x, x + n);
    const double inv = 1.0 / sqrt(nrm);
    for (auto& v : h) v *= inv;
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(L->V, h.data(), n * 8, cudaMemcpyHostToDevice, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    L->started = true;
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_iterate(blqh_lanczos* L, int* steps_done) {
  if (!L) return BLQH_ERR_ARG;
  try {
    cudaSetDevice(L->ctx->device);
    iterate_impl(L);
  } catch (const BlqhError& e) {
    return e.code;
  }
  if (const int rc = blocked_error(L->ctx, L->M)) return rc;
  if (steps_done) *steps_done = L->steps;
  return BLQH_OK;
}

int blqh_lanczos_coeffs(blqh_lanczos* L, double* alpha, double* beta) {
  if (!L) return BLQH_ERR_ARG;
  if (!L->iterated) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_coeffs: call blqh_lanczos_iterate first");
    return BLQH_ERR_STATE;
  }
  blqh_ctx* ctx = L->ctx;
  try {
    const int m = L->steps;
    if (alpha) BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(alpha, L->S.alpha, m * 8, cudaMemcpyDeviceToHost, ctx->stream));
    if (beta) {
      BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(beta, L->S.beta, (m + 1) * 8, cudaMemcpyDeviceToHost, ctx->stream));
      BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      beta[0] = 1.0;
    }
    BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_eig(blqh_lanczos* L, double* eigenvalues, double* psi0) {
  if (!L) return BLQH_ERR_ARG;
  if (!L->iterated || L->steps < 1) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_eig: call blqh_lanczos_iterate first");
    return BLQH_ERR_STATE;
  }
  blqh_ctx* ctx = L->ctx;
  try {
    const int m = L->steps;
    const int lv = tri_smem(L, 2) > 0 ? 2 : 0;
    k_tri_all<<<m, 32, tri_smem(L, lv), ctx->stream>>>(L->S.alpha, L->S.beta, m, L->work + 6 * L->mmax, lv);
    k_tri_vec<<<1, 32, tri_smem(L, 8), ctx->stream>>>(L->S.alpha, L->S.beta, m, L->work + 6 * L->mmax, L->y,
                                                      L->work, tri_smem(L, 8) > 0);
    BLQH_TRY_CUDA(ctx, cudaGetLastError());
    count_launch(ctx, TM_MISC, 2);
    if (eigenvalues)
      BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(eigenvalues, L->work + 6 * L->mmax, m * 8, cudaMemcpyDeviceToHost, ctx->stream));
    if (psi0) BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(psi0, L->y, m * 8, cudaMemcpyDeviceToHost, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_ritz_vector(blqh_lanczos* L, double* psi) {
  if (!L) return BLQH_ERR_ARG;
  if (!L->iterated || L->steps < 1) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_ritz_vector: call blqh_lanczos_iterate first");
    return BLQH_ERR_STATE;
  }
  blqh_ctx* ctx = L->ctx;
  try {
    ritz_impl(L);
    if (psi)
      BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(psi, L->psi, L->dim * L->vw * 8, cudaMemcpyDeviceToHost, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_rayleigh(blqh_lanczos* L, double* energy) {
  if (!L || !energy) return BLQH_ERR_ARG;
  if (!L->have_psi) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_rayleigh: call blqh_lanczos_ritz_vector first");
    return BLQH_ERR_STATE;
  }
  try {
    *energy = rq_stored(L, L->psi);
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_rayleigh_conj(blqh_lanczos* L, const blqh_basis* b, const blqh_params* p, double* energy) {
  if (!L || !energy || (!b != !p)) return BLQH_ERR_ARG;
  if (!L->have_psi) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_rayleigh_conj: call blqh_lanczos_ritz_vector first");
    return BLQH_ERR_STATE;
  }
  if (b && (b->model != BLQH_MODEL_SPINLESS || b->dim != L->dim)) {
    set_error(L->ctx, BLQH_ERR_ARG, "blqh_lanczos_rayleigh_conj: spinless basis of the matrix's sector expected");
    return BLQH_ERR_ARG;
  }
  blqh_ctx* ctx = L->ctx;
  double* xc = nullptr;
  int rc = BLQH_OK;
  try {
    const int64_t n = L->dim * L->vw;
    xc = dalloc<double>(ctx, n);
    k_conj<<<grid_for(ctx, n, 256, 8), 256, 0, ctx->stream>>>(L->psi, xc, n, L->cplx);
    BLQH_TRY_CUDA(ctx, cudaGetLastError());
    count_launch(ctx, TM_MISC);
    *energy = b ? rayleigh_regen_impl(ctx, b, *p, xc, L->cplx != 0) : rq_stored(L, xc);
  } catch (const BlqhError& e) {
    rc = e.code;
  }
  dev_free(xc);
  return rc;
}

int blqh_lanczos_rayleigh_fp64(blqh_lanczos* L, const blqh_basis* b, const blqh_params* p, double* energy) {
  if (!L || !b || !p || !energy) return BLQH_ERR_ARG;
  if (!L->have_psi) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_rayleigh_fp64: call blqh_lanczos_ritz_vector first");
    return BLQH_ERR_STATE;
  }
  if (b->model != BLQH_MODEL_SPINLESS) {
    set_error(L->ctx, BLQH_ERR_ARG, "blqh_lanczos_rayleigh_fp64: spinless bases only (use blqh_lanczos_rayleigh)");
    return BLQH_ERR_ARG;
  }
  if (b->dim != L->dim) {
    set_error(L->ctx, BLQH_ERR_ARG, "blqh_lanczos_rayleigh_fp64: basis does not match the matrix");
    return BLQH_ERR_ARG;
  }
  try {
    if (L->M->d_res && L->xs && !regen_forced()) *energy = rayleigh_res_impl(L);
    else *energy = rayleigh_regen_impl(L->ctx, b, *p, L->psi, L->cplx != 0);
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_destroy(blqh_lanczos* L) {
  free_lanczos(L);
  return BLQH_OK;
}

int blqh_start_vector(uint64_t seed, int rng, int64_t dim, int is_complex, double* out) {
  if (!out || dim < 0 || (rng != 0 && rng != 1)) return BLQH_ERR_ARG;
  fill_start(seed, rng, dim, is_complex, out);
  return BLQH_OK;
}

int blqh_ground_state(blqh_ctx* ctx, const blqh_sector* s, const blqh_params* p, int prec,
                      const blqh_lanczos_opts* o, const double* start, double* psi, blqh_result* out) {
  if (!ctx || !s || !p || !o || !out) return BLQH_ERR_ARG;
  blqh_basis* B = nullptr;
  blqh_csr* M = nullptr;
  blqh_lanczos* L = nullptr;
  int rc = blqh_basis_build(ctx, s, &B);
  if (rc == BLQH_OK) rc = blqh_hamil_build(ctx, B, p, prec, &M);
  if (rc == BLQH_OK) rc = blqh_lanczos_create(ctx, M, o, &L);
  if (rc == BLQH_OK && start) rc = blqh_lanczos_set_start(L, start);
  int steps = 0;
  if (rc == BLQH_OK) rc = blqh_lanczos_iterate(L, &steps);
  if (rc == BLQH_OK) rc = blqh_lanczos_ritz_vector(L, psi);
  double e = 0;
  if (rc == BLQH_OK) {
    if (prec == BLQH_VAL_FP64) rc = blqh_lanczos_rayleigh(L, &e);
    else rc = blqh_lanczos_rayleigh_fp64(L, B, p, &e);
  }
  if (rc == BLQH_OK) {
    double r0 = 0;
    cudaMemcpy(&r0, L->work + 6 * L->mmax, 8, cudaMemcpyDeviceToHost);
    out->energy = e;
    out->ritz0 = r0;
    out->steps = steps;
    out->dim = B->dim;
    out->nnz = M->nnz;
  }
  blqh_lanczos_destroy(L);
  blqh_csr_destroy(M);
  blqh_basis_destroy(B);
  return rc;
}

int blqh_lanczos_observables(blqh_lanczos* L, const blqh_basis* b, double* sz, double* sx, double* occ) {
  if (!L || !b) return BLQH_ERR_ARG;
  if (!L->have_psi) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_observables: call blqh_lanczos_ritz_vector first");
    return BLQH_ERR_STATE;
  }
  if (b->dim != L->dim) {
    set_error(L->ctx, BLQH_ERR_ARG, "blqh_lanczos_observables: basis does not match the Hamiltonian");
    return BLQH_ERR_ARG;
  }
  try {
    observables_impl(L->ctx, b, L->psi, L->cplx, sz, sx, occ);
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_rayleigh_fp64_spin(blqh_lanczos* L, const blqh_basis* b, const blqh_params_spin* p,
                                    double* energy) {
  if (!L || !b || !p || !energy) return BLQH_ERR_ARG;
  if (!L->have_psi) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_rayleigh_fp64_spin: call blqh_lanczos_ritz_vector first");
    return BLQH_ERR_STATE;
  }
  if (b->model != BLQH_MODEL_SPINFUL || b->dim != L->dim) {
    set_error(L->ctx, BLQH_ERR_ARG, "blqh_lanczos_rayleigh_fp64_spin: spinful basis of the matrix's sector expected");
    return BLQH_ERR_ARG;
  }
  try {
    *energy = spin_rayleigh_regen_impl(L->ctx, b, *p, L->psi);
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_lanczos_observables_spin(blqh_lanczos* L, const blqh_basis* b, double* out) {
  if (!L || !b || !out) return BLQH_ERR_ARG;
  if (!L->have_psi) {
    set_error(L->ctx, BLQH_ERR_STATE, "blqh_lanczos_observables_spin: call blqh_lanczos_ritz_vector first");
    return BLQH_ERR_STATE;
  }
  if (b->model != BLQH_MODEL_SPINFUL || b->dim != L->dim) {
    set_error(L->ctx, BLQH_ERR_ARG, "blqh_lanczos_observables_spin: spinful basis of the matrix's sector expected");
    return BLQH_ERR_ARG;
  }
  try {
    spin_observables_impl(L->ctx, b, L->psi, L->cplx, out);
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_debug_lanczos_product(blqh_lanczos* L, double* x, double* y) {
  if (!L || !x || !y) return BLQH_ERR_ARG;
  blqh_ctx* ctx = L->ctx;
  try {
    const int64_t n = L->dim * L->vw;
    const int m = L->iterated ? L->steps : 0;
    if (!L->started) {
      set_error(ctx, BLQH_ERR_STATE, "blqh_debug_lanczos_product: no start vector yet");
      return BLQH_ERR_STATE;
    }
    const double* v = L->V + (int64_t)m * n;
    spmv_dev(ctx, L->M, v, L->w, nullptr, nullptr, nullptr, L->xs, m > 0, &L->fx, L->xq, L->xe, L->pmax);
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(x, v, n * 8, cudaMemcpyDeviceToHost, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaMemcpyAsync(y, L->w, n * 8, cudaMemcpyDeviceToHost, ctx->stream));
    BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_debug_spmv_layout(const blqh_csr* M) {
  if (!M) return -1;
  return M->blk_state > 0 ? (M->blk_dict > 0 ? 2 : 1) : 0;
}

}  // extern "C"
