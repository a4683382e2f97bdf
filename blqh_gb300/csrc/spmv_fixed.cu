// SpMV of complex FP64 matrices in fixed point (y = H x - b xprev, the Lanczos
// product of Mat::operator*, BLQH_without_spin/matrix.cpp:244-267).
//
// The FP64 row kernel issues four FP64 FMAs per nonzero and ten FP64 additions per
// row on a pipe of ~1.6 lane operations per clock per SM: that pipe, not memory,
// sets its time. Here both operands are integers, split once: the matrix per row (57
// bits below the row's largest off-diagonal entry; the diagonal stays FP64 and
// apart), the vector on the scale of its largest entry (|x| <= 2^xe, at most 4 times
// that entry),
//   v = (v1 2^29 + v0) 2^(E - 56),   |v1|, |v0| <= 2^28,
//   x = (x1 2^29 + x0) 2^(xe - 59),  |x1| <= 2^30, |x0| <= 2^28,
// and a row's sum is exact integer arithmetic: four IMAD.WIDE (27 lanes per clock
// per SM) per real product into three 64-bit sums, folded into 128 bits every
// eight nonzeros (the largest sum, of 2 x 8 cross products below 1.25 x 2^58, stays
// below 2^63), one conversion to FP64 per row. What is lost is the operands'
// rounding, 2^-57 of the row's and 2^-58 of the vector's largest entry: entries far
// below those keep fewer bits than FP64's 53, but a row's sum is not rounded at every
// addition. Error against extended precision, root mean square over rows, Krylov
// vectors of 79 to 100,141 states: 0.27 to 0.66 of the FP64 kernel's; rows of states
// where the vector is zero, which leave the FP64 diagonal term out: 0.28 to 0.36
// (tests/test_fixed_product.py; with the unit at 2^-59 of the vector's norm the latter
// were 0.41 to 1.003, growing with the number of states).
//
// The split matrix takes 16 bytes per nonzero next to the CSR values. What is left
// is the latency of the column, then the gather behind it (long-scoreboard stalls,
// 12 of 20 cycles per issue; DRAM 46 %), so a lane has eight columns, then four
// values and four gathers in flight. Measured (one GB300): 60,096 rows,
// 1.54e7 nonzeros 212 -> 84 us; 100,141 rows, 2.4e7 nonzeros 318 -> 119 us;
// 16,024 rows, 2.1e6 nonzeros 54 -> 22 us.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "blqh_internal.h"
#include "krylov.cuh"
#include "gs_fixed.cuh"

namespace {

// Up to here one block splits a vector in less than the ~4 us of a second launch (8 entries a thread).
constexpr int64_t FIX_SHORT = 8192;

// Row exponents, split off-diagonal values and the diagonal: one warp per row. The
// exponent is raised until the row's sum of |q| stays below 2^67 (rows of up to 512
// nonzeros always do), so that a product with |x| <= 2^59 units stays below 2^127. A row
// with an infinite or NaN entry, which has no integers, gets a NaN diagonal: its
// product is then NaN.
__global__ void __launch_bounds__(256) k_fix_matrix(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                                                    const double2* __restrict__ val, int64_t dim,
                                                    int4* __restrict__ qv, int* __restrict__ qe,
                                                    double2* __restrict__ diag) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < dim; r += warps) {
    const int64_t s = rp[r], e = rp[r + 1];
    unsigned hw = 0;
    bool has = false;
    for (int64_t k = s + lane; k < e; k += 32) {
      const double2 v = val[k];
      if (col[k] == r) {
        diag[r] = v;
        has = true;
      } else {
        hw = max(hw, max(abs_high_word(v.x), abs_high_word(v.y)));
      }
    }
    hw = __reduce_max_sync(0xffffffffu, hw);
    has = __any_sync(0xffffffffu, has);
    int E = word_exponent(hw);
    for (;; E++) {
      long long sum = 0;  // of |q| / 2^29, rounded up
      for (int64_t k = s + lane; k < e; k += 32) {
        int4 q = make_int4(0, 0, 0, 0);
        if (col[k] != r) {
          const double2 v = val[k];
          quantize(v.x, E, q.x, q.y);
          quantize(v.y, E, q.z, q.w);
          sum += abs(q.x) + abs(q.z) + 2;
        }
        qv[k] = q;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (sum <= 1LL << 38) break;
    }
    if (lane == 0) {
      qe[r] = E;
      if (!has) diag[r] = make_double2(0.0, 0.0);
      if (word_exponent(hw) == 1024) diag[r].x = diag[r].y = __longlong_as_double(0x7FF8000000000000LL);
    }
  }
}

// x in the vector's fixed point, for products whose previous kernel did not leave it:
// the largest entry's high word (*xmax zero before), then the entries and their scale.
__global__ void __launch_bounds__(256) k_fix_max(const double* __restrict__ x, unsigned* xmax, int64_t n,
                                                 const int* stop) {
  if (stop && *stop) return;
  __shared__ unsigned red[8];
  unsigned hw = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    hw = max(hw, abs_high_word(x[i]));
  hw = block_max(hw, red);
  if (threadIdx.x == 0) atomicMax(xmax, hw);
}
// Both in one block, for short vectors: one launch where they are two and a memset.
__global__ void __launch_bounds__(1024) k_fix_short(const double* __restrict__ x, int2* __restrict__ xq, int* xe,
                                                    int n, const int* stop) {
  if (stop && *stop) return;
  __shared__ unsigned red[32];
  unsigned hw = 0;
  for (int i = threadIdx.x; i < n; i += 1024) hw = max(hw, abs_high_word(x[i]));
  const int e = min(word_exponent(block_max(hw, red)) + 1, 0);
  if (threadIdx.x == 0) *xe = e;
  for (int i = threadIdx.x; i < n; i += 1024) xq[i] = fix_scaled(x[i], e);
}
__global__ void k_fix_vector(const double* __restrict__ x, int2* __restrict__ xq, int* xe, const unsigned* xmax,
                             int64_t n, const int* stop) {
  if (stop && *stop) return;
  const int e = min(word_exponent(*xmax) + 1, 0);
  if (blockIdx.x == 0 && threadIdx.x == 0) *xe = e;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    xq[i] = fix_scaled(x[i], e);
}

// LPR lanes per row. The real and imaginary sums are reduced together: after the
// first exchange the lower half of a row's lanes carries the real part, the upper
// half the imaginary part.
template <int LPR>
__global__ void __launch_bounds__(256, 3) k_spmv_fixed(const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                                                    const int4* __restrict__ qv, const int* __restrict__ qe,
                                                    const double2* __restrict__ diag, const int4* xq,
                                                    const int* __restrict__ xe,
                                                    const double2* x, double2* __restrict__ y, int64_t dim,
                                                    const double* bptr, const double2* xprev, const int* stop) {
  if (stop && *stop) return;
  const int lane = threadIdx.x & 31;
  constexpr int GPW = 32 / LPR;
  const int gi = lane / LPR, sub = lane % LPR;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const double b = bptr ? *bptr : 0.0;
  for (int64_t rb = warp * GPW; rb < dim; rb += nwarps * GPW) {  // the same rounds for every lane
    const int64_t r = rb + gi;
    const bool ok = r < dim;
    const int64_t s = ok ? __ldg(rp + r) : 0;
    const int len = ok ? (int)(__ldg(rp + r + 1) - s) : 0;
    const int4* vp = qv + s;
    const int32_t* cp = col + s;
    Acc128 re{0, 0}, im{0, 0};
    // eight nonzeros per lane at a time: the eight columns, then values and
    // gathers of four; `full`: none of them past the row's end
    auto group = [&](int k, auto full) {
      constexpr bool F = decltype(full)::value;
      int c[8];
#pragma unroll
      for (int u = 0; u < 8; u++) c[u] = F || k + u * LPR < len ? __ldcs(cp + k + u * LPR) : 0;
      long long sr[3] = {0, 0, 0}, si[3] = {0, 0, 0};
#pragma unroll
      for (int h = 0; h < 8; h += 4) {
        int4 v[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          v[u] = F || k + (h + u) * LPR < len ? __ldcs(vp + k + (h + u) * LPR) : make_int4(0, 0, 0, 0);
          g[u] = __ldg(xq + c[h + u]);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
          fx_add(sr, v[u].x, v[u].y, g[u].x, g[u].y);
          fx_add(sr, -v[u].z, -v[u].w, g[u].z, g[u].w);
          fx_add(si, v[u].x, v[u].y, g[u].z, g[u].w);
          fx_add(si, v[u].z, v[u].w, g[u].x, g[u].y);
        }
      }
      re.fold(sr);
      im.fold(si);
    };
    int k = sub;
    for (; k + 7 * LPR < len; k += 8 * LPR) group(k, std::true_type());
    if (k < len) group(k, std::false_type());
    const bool upper = sub >= LPR / 2;
    Acc128 a = upper ? im : re;
    const Acc128 o = upper ? re : im;
    a.add(__shfl_xor_sync(0xffffffffu, o.lo, LPR / 2), __shfl_xor_sync(0xffffffffu, o.hi, LPR / 2));
#pragma unroll
    for (int d = LPR / 4; d > 0; d >>= 1)
      a.add(__shfl_xor_sync(0xffffffffu, a.lo, d), __shfl_xor_sync(0xffffffffu, a.hi, d));
    // 2^(E - 56) of the matrix times 2^(xe - 59) of the vector
    const double part = ok ? fx_to_double(a.hi, a.lo, __ldg(qe + r) + __ldg(xe) - 115) : 0.0;
    const double other = __shfl_xor_sync(0xffffffffu, part, LPR / 2);
    if (ok && sub == 0) {
      const double2 d = __ldg(diag + r), xr = x[r];
      double2 w = make_double2(part + (d.x * xr.x - d.y * xr.y), other + (d.x * xr.y + d.y * xr.x));
      if (xprev) {
        const double2 p = xprev[r];
        w.x -= b * p.x;
        w.y -= b * p.y;
      }
      y[r] = w;
    }
  }
}

}  // namespace

// The split copy of a complex FP64 matrix; false (and the FP64 kernel stays) without
// room for it or with BLQH_SPMV_FIXED=0.
bool fixed_prepare(blqh_ctx* ctx, const blqh_csr* M, FixedMatrix* F) {
  if (!M->is_complex || M->precision != BLQH_VAL_FP64) return false;
  const char* env = getenv("BLQH_SPMV_FIXED");
  if (env && env[0] == '0') return false;
  try {
    F->val = dev_alloc(ctx, std::max<int64_t>(1, M->nnz) * sizeof(int4));
    F->row_exp = dalloc<int>(ctx, M->dim);
    F->diag = dalloc<double>(ctx, 2 * M->dim);
  } catch (const BlqhError& e) {
    if (e.code != BLQH_ERR_NOMEM) throw;
    fixed_release(F);
    ctx->last_error.clear();
    return false;
  }
  TimerScope ts(ctx, TM_MISC);
  k_fix_matrix<<<grid_for(ctx, M->dim * 32, 256, 16), 256, 0, ctx->stream>>>(
      M->d_row_ptr, M->d_col, reinterpret_cast<const double2*>(M->d_val), M->dim, static_cast<int4*>(F->val), F->row_exp,
      reinterpret_cast<double2*>(F->diag));
  BLQH_TRY_CUDA(ctx, cudaGetLastError());
  count_launch(ctx, TM_MISC);
  return true;
}

void fixed_release(FixedMatrix* F) {
  dev_free(F->val);
  dev_free(F->row_exp);
  dev_free(F->diag);
  *F = FixedMatrix{};
}

// x (|x| <= 1, as Krylov vectors are) in fixed point; xmax: scratch.
void fixed_vector(blqh_ctx* ctx, const double* x, int2* xq, int* xe, unsigned* xmax, int64_t n, const int* stop) {
  TimerScope tm(ctx, TM_MISC);
  if (n <= FIX_SHORT) {
    k_fix_short<<<1, 1024, 0, ctx->stream>>>(x, xq, xe, (int)n, stop);
    BLQH_TRY_CUDA(ctx, cudaGetLastError());
    count_launch(ctx, TM_MISC);
    return;
  }
  const int grid = grid_for(ctx, n, 256, 8);
  BLQH_TRY_CUDA(ctx, cudaMemsetAsync(xmax, 0, sizeof(unsigned), ctx->stream));
  k_fix_max<<<grid, 256, 0, ctx->stream>>>(x, xmax, n, stop);
  k_fix_vector<<<grid, 256, 0, ctx->stream>>>(x, xq, xe, xmax, n, stop);
  BLQH_TRY_CUDA(ctx, cudaGetLastError());
  count_launch(ctx, TM_MISC, 2);
}

// y = H x - b xprev; xq, xe: x in fixed point.
void fixed_spmv(blqh_ctx* ctx, const blqh_csr* M, const FixedMatrix& F, const double* x, const int2* xq, const int* xe,
                double* y, const double* bptr, const double* xprev, const int* stop) {
  // 8 lanes per row (four rows per warp): 84 us at 60,096 rows of 256 nonzeros, against
  // 92 with 4 lanes, 95 with 16 and 121 with 32 (longer reductions per row)
  constexpr int LPR = 8;
  const int64_t blocks = std::min<int64_t>((M->dim * LPR + 255) / 256, (int64_t)ctx->num_sms * 16);
  k_spmv_fixed<LPR><<<(int)std::max<int64_t>(1, blocks), 256, 0, ctx->stream>>>(
      M->d_row_ptr, M->d_col, static_cast<const int4*>(F.val), F.row_exp, reinterpret_cast<const double2*>(F.diag),
      reinterpret_cast<const int4*>(xq), xe,
      reinterpret_cast<const double2*>(x), reinterpret_cast<double2*>(y), M->dim, bptr,
      reinterpret_cast<const double2*>(xprev), stop);
}
