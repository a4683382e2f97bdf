// K9: batched sweep. Many (sector, parameter point) instances of uneven
// dimension advance in ONE persistent kernel: each thread block takes the next
// instance from a device work queue (ordered by decreasing cost), runs its
// whole Lanczos recurrence with full FP64 reorthogonalization, solves its
// tridiagonal and forms its ground state, then takes the next instance. The
// instance's SpMV input vector lives in shared memory (as FP32 pairs for the
// double-float product when the values are FP32, as FP64 otherwise), so the
// gathers of the SpMV never leave the SM; the Krylov basis streams from HBM.
// No block waits for another block: there is no grid barrier and no spin.
//
// Replaces the sweep loops of the reference's drivers (BLQH_without_spin/
// main.cpp:77-115 over momentum sectors, :134-181 over layer distance), which
// call basis::init, lhamil::set_hamil, coeff_explicit_update, diag,
// eigenstates_reconstruction and ground_state_energy once per point
// (lanczos_hamiltonian.cpp:87-656). Per step: the three-term step (remove the
// components along v_j and v_{j-1}), then one full classical Gram-Schmidt
// pass against every stored vector, and a further pass when the norm fell
// below 1/sqrt(2) of its value after the three-term step (the
// Daniel-Gragg-Kaufman-Stewart criterion). Real instances run the pass in FP64, in
// a fixed order of operations (their ground states can be degenerate, see
// gs_ordered.cuh, and then depend on it); complex instances take it on fixed-point
// planes of the Krylov basis (gs_fixed.cuh), one exponent per vector (57 bits below its
// largest entry): exact integer dots (error against extended precision, random vectors
// of 79 to 100,141 complex entries: 0.18 to 0.42 of the FP64 dots'), and the correction
// in FP32 while every coefficient is below 2^-36 |w|. The FP64 pass of a complex
// instance took the SM's FP64 pipe 8 FMAs per entry and vector; 96 instances of 5,940
// states, 150 steps: 348 -> 134 ms. The lowest Ritz pair comes from Sturm
// multisection and inverse iteration; the finisher is the FP64 regenerated Rayleigh
// quotient for FP32 values, the stored FP64 CSR otherwise.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <tuple>
#include <vector>

#include "krylov.cuh"
#include "gs_fixed.cuh"
#include "sector.cuh"

namespace {

// One instance as the persistent kernel sees it.
struct BInst {
  const int64_t* rp;
  const int32_t* col;
  const void* val;
  int64_t dim;
  int cplx, fp32, xsmem;
  int number;     // position in the caller's list (start-vector stream)
  double* V;      // [(lam + 1) * N], N = dim * (cplx ? 2 : 1)
  double* w;      // [N]
  double* psi;    // [N]
  double* ab;     // alpha [lam], beta [lam + 1] (beta[0] = 0)
  double* res;    // [5]: energy, lowest Ritz value, residual estimate, steps, repeated Gram-Schmidt passes
  double* xg;     // [N] staging of the SpMV input in global memory when it does not fit shared memory
  // complex: fixed-point planes of V [(lam + 1) * NP] and of w [NP], NP = N rounded up to 4 (null: FP64 pass)
  int* q1;
  int* q0;
};

constexpr int RED = 66;  // doubles of the block-reduction area

// Shared-memory layout (doubles): red | hs, h2 [2 (lam+1)] | ta [lam] | tb [lam+1] | ys [lam] |
// tri work [6 lam] | scal [8] | x area (rounded to 32 bytes: the x area takes 16-byte loads).
__host__ __device__ inline int batch_fixed_doubles(int lam) {
  return (RED + 4 * (lam + 1) + 9 * lam + 1 + 8 + 3) / 4 * 4;
}

// Per-instance device storage, in doubles from the instance's block (each array 256-byte aligned).
struct Lay {
  size_t V, w, psi, ab, xg, total;
};
inline Lay instance_layout(int64_t N, int lam, bool xsmem) {
  auto up = [](size_t v) { return (v + 31) / 32 * 32; };
  Lay L;
  L.V = 0;
  L.w = up((size_t)N * (lam + 1));
  L.psi = up(L.w + N);
  L.ab = up(L.psi + N);
  L.xg = up(L.ab + 2 * lam + 1);
  L.total = up(L.xg + (xsmem ? 0 : (size_t)N));
  return L;
}
// One plane of a complex instance: w's after the lam + 1 vectors' (ints, 256-byte aligned).
inline size_t plane_ints(int64_t N, int lam) { return ((size_t)(lam + 2) * (size_t)((N + 3) / 4 * 4) + 63) / 64 * 64; }

template <int NT>
__device__ __forceinline__ void block_sum2(double& a, double& b, double* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane == 0) {
    red[2 * wid] = a;
    red[2 * wid + 1] = b;
  }
  __syncthreads();
  if (wid == 0) {
    double x = lane < NT / 32 ? red[2 * lane] : 0.0, y = lane < NT / 32 ? red[2 * lane + 1] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      x += __shfl_xor_sync(0xffffffffu, x, o);
      y += __shfl_xor_sync(0xffffffffu, y, o);
    }
    if (lane == 0) {
      red[64] = x;
      red[65] = y;
    }
  }
  __syncthreads();
  a = red[64];
  b = red[65];
}

// Calls use(i, load(i)) for this thread's i < n in ascending order, U loads in flight
// (stores in `use` would otherwise order every load behind the previous entry's).
template <int NT, int U, class L, class F>
__device__ __forceinline__ void sweep(int64_t n_, L load, F use) {
  const int n = (int)n_;
  int i = threadIdx.x;
  for (; i + (U - 1) * NT < n; i += U * NT) {
    decltype(load(i)) r[U];
#pragma unroll
    for (int u = 0; u < U; u++) r[u] = load(i + u * NT);
#pragma unroll
    for (int u = 0; u < U; u++) use(i + u * NT, r[u]);
  }
#pragma unroll 1
  for (; i < n; i += NT) use(i, load(i));
}

template <bool CPLX, bool F32>
struct ValT;
template <>
struct ValT<false, false> {
  using T = double;
};
template <>
struct ValT<true, false> {
  using T = double2;
};
template <>
struct ValT<false, true> {
  using T = float;
};
template <>
struct ValT<true, true> {
  using T = float2;
};

// w = H x (rq = false), or the partial Re <x, H x> of this thread (rq = true,
// FP64 values only). x: FP32 pairs (hi, lo) per double when F32 (complex entries as
// (re hi, im hi, re lo, im lo), so that both parts go through packed FP32 operations
// at once), FP64 otherwise; in shared or global memory. F32: w receives the unevaluated
// (hi, lo) pair of every component (same 8 bytes); converting here would cost
// every lane of a row group an FP64 instruction, so run_instance converts them
// lane-parallel.
// A block is all its SM runs, so the matrix stream's latency shows: each lane keeps
// the next BS nonzeros (of its row, or the first ones of its next row) in flight
// behind the ones it works on. Sums are in column order per lane as without it.
template <int NT, int LPR, bool CPLX, bool F32>
__device__ __forceinline__ double bspmv(const BInst& I, const void* __restrict__ x, double* __restrict__ w,
                                        bool rq) {
  using VT = typename ValT<CPLX, F32>::T;
  constexpr int NG = NT / LPR;
  constexpr int BS = 8;
  const int grp = threadIdx.x / LPR, sub = threadIdx.x % LPR;
  const VT* __restrict__ val = reinterpret_cast<const VT*>(I.val);
  double dot = 0.0;
  auto range = [&](int64_t r, int64_t& s, int64_t& e) {
    const bool ok = r < I.dim;
    s = ok ? __ldg(I.rp + r) : 0;
    e = ok ? __ldg(I.rp + r + 1) : 0;
  };
  int32_t cc[BS];
  VT vv[BS];
  auto load = [&](int32_t (&c)[BS], VT (&v)[BS], int64_t k, int64_t e) {
#pragma unroll
    for (int u = 0; u < BS; u++) {
      c[u] = 0;
      v[u] = VT{};
      if (k + u * LPR < e) {
        c[u] = __ldg(I.col + k + u * LPR);
        v[u] = __ldg(val + k + u * LPR);
      }
    }
  };
  int64_t s, e, s1, e1;  // this row's range and the next one's
  range(grp, s, e);
  range(grp + NG, s1, e1);
  load(cc, vv, s + sub, e);
  for (int64_t rb = 0; rb < I.dim; rb += NG) {
    const int64_t r = rb + grp;
    const bool ok = r < I.dim;
    int64_t s2, e2;
    range(r + 2 * NG, s2, e2);
    float rh = 0.f, rl = 0.f, ih = 0.f, il = 0.f;
    double ar = 0.0, ai = 0.0;
    f32x2 ah = 0, al = 0, bh = 0, bl = 0;  // F32 complex: sums of Re v (re, im) x and of (Im v, -Im v) (re, im) x
    int64_t k = s + sub;
    for (;;) {
      const bool more = k + BS * LPR < e;
      int32_t cn[BS];
      VT vn[BS];
      load(cn, vn, more ? k + BS * LPR : s1 + sub, more ? e : e1);
#pragma unroll
      for (int u = 0; u < BS; u++) {
        if (k + u * LPR < e) {
          const int32_t c = cc[u];
          if constexpr (F32 && CPLX) {
            const ulonglong2 xv = reinterpret_cast<const ulonglong2*>(x)[c];
            df_add_prod2(ah, al, pack2(vv[u].x, vv[u].x), xv.x, xv.y);
            df_add_prod2(bh, bl, pack2(vv[u].y, -vv[u].y), xv.x, xv.y);
          } else if constexpr (F32) {
            const float2 xv = reinterpret_cast<const float2*>(x)[c];
            df_add_prod(rh, rl, vv[u], xv.x, xv.y);
          } else if constexpr (CPLX) {
            const double2 xv = reinterpret_cast<const double2*>(x)[c];
            ar += vv[u].x * xv.x - vv[u].y * xv.y;
            ai += vv[u].x * xv.y + vv[u].y * xv.x;
          } else {
            ar += vv[u] * reinterpret_cast<const double*>(x)[c];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < BS; u++) {
        cc[u] = cn[u];
        vv[u] = vn[u];
      }
      if (!more) break;
      k += BS * LPR;
    }
    __syncwarp();
    if (F32 && CPLX) {  // re = a.re + b.im (-Im v Im x), im = a.im + b.re
      const float2 a = unpack2(ah), b = unpack2(al), c = unpack2(bh), d = unpack2(bl);
      rh = a.x;
      rl = b.x;
      ih = a.y;
      il = b.y;
      df_add(rh, rl, c.y, d.y);
      df_add(ih, il, c.x, d.x);
    }
    if (F32) {
      df_seg_reduce<LPR>(rh, rl);
      if (CPLX) df_seg_reduce<LPR>(ih, il);
      if (ok && sub == 0) {
        float2* wp = reinterpret_cast<float2*>(w);
        if (CPLX) {
          wp[2 * r] = make_float2(rh, rl);
          wp[2 * r + 1] = make_float2(ih, il);
        } else {
          wp[r] = make_float2(rh, rl);
        }
      }
    } else {
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) {
        ar += __shfl_xor_sync(0xffffffffu, ar, o, LPR);
        if (CPLX) ai += __shfl_xor_sync(0xffffffffu, ai, o, LPR);
      }
      if (ok && sub == 0) {
        if (rq) {
          if (CPLX) {
            const double2 p = reinterpret_cast<const double2*>(x)[r];
            dot += p.x * ar + p.y * ai;
          } else {
            dot += reinterpret_cast<const double*>(x)[r] * ar;
          }
        } else if (CPLX) {
          reinterpret_cast<double2*>(w)[r] = make_double2(ar, ai);
        } else {
          w[r] = ar;
        }
      }
    }
    s = s1;
    e = e1;
    s1 = s2;
    e1 = e2;
  }
  return dot;
}

// h[k] = <V_k, w> for k < nk (complex: conj(V_k) w), one warp per vector.
// Two independent accumulator sets per lane keep two loads and FMA chains in flight.
template <int NT, bool CPLX>
__device__ __forceinline__ void cgs_dots(const double* __restrict__ V, int64_t N, int nk,
                                         const double* __restrict__ w, double* h) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int k = wid; k < nk; k += NT / 32) {
    const double* vk = V + (int64_t)k * N;
    double sr = 0.0, si = 0.0, tr = 0.0, ti = 0.0;
    if (CPLX) {
      const double2* a2 = reinterpret_cast<const double2*>(vk);
      const double2* b2 = reinterpret_cast<const double2*>(w);
      const int64_t n2 = N / 2;
      int64_t i = lane;
#pragma unroll 2
      for (; i + 32 < n2; i += 64) {
        const double2 a = a2[i], b = b2[i], c = a2[i + 32], d = b2[i + 32];
        sr += a.x * b.x + a.y * b.y;
        si += a.x * b.y - a.y * b.x;
        tr += c.x * d.x + c.y * d.y;
        ti += c.x * d.y - c.y * d.x;
      }
      if (i < n2) {
        const double2 a = a2[i], b = b2[i];
        sr += a.x * b.x + a.y * b.y;
        si += a.x * b.y - a.y * b.x;
      }
    } else {
      int64_t i = lane;
#pragma unroll 4
      for (; i + 32 < N; i += 64) {
        sr += vk[i] * w[i];
        tr += vk[i + 32] * w[i + 32];
      }
      if (i < N) sr += vk[i] * w[i];
    }
    sr += tr;
    si += ti;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sr += __shfl_xor_sync(0xffffffffu, sr, o);
      si += __shfl_xor_sync(0xffffffffu, si, o);
    }
    if (lane == 0) {
      h[2 * k] = sr;
      h[2 * k + 1] = si;
    }
  }
}

// w -= sum_k V_k h_k; returns this thread's partial |w|^2.
template <int NT, bool CPLX>
__device__ __forceinline__ double cgs_update(const double* __restrict__ V, int64_t N, int nk, const double* h,
                                             double* __restrict__ w) {
  double nn = 0.0;
  if (CPLX) {
    for (int64_t i = threadIdx.x; i < N / 2; i += NT) {
      double2 acc = reinterpret_cast<double2*>(w)[i];
      double2 bcc = make_double2(0.0, 0.0);
      int k = 0;
      for (; k + 2 <= nk; k += 2) {
        const double2 v = reinterpret_cast<const double2*>(V + (int64_t)k * N)[i];
        const double2 u = reinterpret_cast<const double2*>(V + (int64_t)(k + 1) * N)[i];
        const double hr = h[2 * k], hi = h[2 * k + 1], gr = h[2 * k + 2], gi = h[2 * k + 3];
        acc.x -= hr * v.x - hi * v.y;
        acc.y -= hr * v.y + hi * v.x;
        bcc.x -= gr * u.x - gi * u.y;
        bcc.y -= gr * u.y + gi * u.x;
      }
      if (k < nk) {
        const double2 v = reinterpret_cast<const double2*>(V + (int64_t)k * N)[i];
        const double hr = h[2 * k], hi = h[2 * k + 1];
        acc.x -= hr * v.x - hi * v.y;
        acc.y -= hr * v.y + hi * v.x;
      }
      acc.x += bcc.x;
      acc.y += bcc.y;
      reinterpret_cast<double2*>(w)[i] = acc;
      nn += acc.x * acc.x + acc.y * acc.y;
    }
  } else {
    for (int64_t i = threadIdx.x; i < N; i += NT) {
      double acc = w[i], bcc = 0.0;
      int k = 0;
      for (; k + 2 <= nk; k += 2) {
        const double v0 = V[(int64_t)k * N + i], v1 = V[(int64_t)(k + 1) * N + i];
        acc -= h[2 * k] * v0;
        bcc -= h[2 * k + 2] * v1;
      }
      if (k < nk) acc -= h[2 * k] * V[(int64_t)k * N + i];
      acc += bcc;
      w[i] = acc;
      nn += acc * acc;
    }
  }
  return nn;
}

// ---- the full pass of complex instances on fixed-point planes --------------------
// Bits that partial sums of an N-entry dot drop at their lower end so that the whole
// of it (N products below 2^114) stays below 2^127: 2^-101 of its largest product
// and less, nothing against the operands' 2^-57.
__device__ __forceinline__ int sum_shift(int64_t N) {
  const int lg = 64 - __clzll(N);
  return lg > 12 ? lg - 12 : 0;
}

// Exponent of the block's largest |x| (in every thread).
template <int NT>
__device__ __forceinline__ int plane_exponent(unsigned hw, double* red) {
  unsigned* ur = reinterpret_cast<unsigned*>(red);
  hw = __reduce_max_sync(0xffffffffu, hw);
  if ((threadIdx.x & 31) == 0) ur[threadIdx.x >> 5] = hw;
  __syncthreads();
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < NT / 32; i++) m = max(m, ur[i]);
  __syncthreads();
  return word_exponent(m);
}

// Planes of x (N entries, FP64, written by this block) with exponent E; zeros up to NP.
template <int NT>
__device__ __forceinline__ void write_planes(const double* x, int64_t N, int64_t NP, int E, int* q1, int* q0) {
  sweep<NT, 4>(
      NP, [&](int i) { return i < N ? x[i] : 0.0; },
      [&](int i, double v) {
        int a, b;
        quantize(v, E, a, b);
        q1[i] = a;
        q0[i] = b;
      });
}

// h[k] = conj(V_k) w from the planes, a warp two vectors at a time (w read once for both).
template <int NT>
__device__ __forceinline__ void cgs_dots_q(const int* __restrict__ q1, const int* __restrict__ q0, int64_t NP,
                                           const int* qe, int nk, const int* w1, const int* w0, int we, double* h) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int n4 = (int)(NP / 4), shift = sum_shift(NP);
  for (int k = 2 * wid; k < nk; k += 2 * (NT / 32)) {
    const int kb = min(k + 1, nk - 1);  // a missing second vector repeats the first
    const int4* a1 = reinterpret_cast<const int4*>(q1 + k * NP);
    const int4* a0 = reinterpret_cast<const int4*>(q0 + k * NP);
    const int4* b1 = reinterpret_cast<const int4*>(q1 + kb * NP);
    const int4* b0 = reinterpret_cast<const int4*>(q0 + kb * NP);
    Acc128 t[4] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};  // (re, im) of both
    auto one = [&](long long (&s)[3], long long (&r)[3], const int4& x1, const int4& x0, const int4& y1,
                   const int4& y0) {  // conj(x) y of two entries
      fx_add(s, x1.x, x0.x, y1.x, y0.x);
      fx_add(s, x1.y, x0.y, y1.y, y0.y);
      fx_add(s, x1.z, x0.z, y1.z, y0.z);
      fx_add(s, x1.w, x0.w, y1.w, y0.w);
      fx_add(r, x1.x, x0.x, y1.y, y0.y);
      fx_add(r, -x1.y, -x0.y, y1.x, y0.x);
      fx_add(r, x1.z, x0.z, y1.w, y0.w);
      fx_add(r, -x1.w, -x0.w, y1.z, y0.z);
    };
    for (int i0 = lane; i0 < n4; i0 += 8 * 32) {  // 32 products per 64-bit sum
      long long s[4][3] = {};
#pragma unroll 2
      for (int u = 0; u < 8; u++) {
        const int i = i0 + 32 * u;
        if (i >= n4) break;
        const int4 x1 = __ldcg(a1 + i), x0 = __ldcg(a0 + i), z1 = __ldcg(b1 + i), z0 = __ldcg(b0 + i);
        const int4 y1 = reinterpret_cast<const int4*>(w1)[i], y0 = reinterpret_cast<const int4*>(w0)[i];
        one(s[0], s[1], x1, x0, y1, y0);
        one(s[2], s[3], z1, z0, y1, y0);
      }
#pragma unroll
      for (int c = 0; c < 4; c++) t[c].fold(s[c], shift);
    }
    const int ea = qe[k] + we - 112 + shift, eb = qe[kb] + we - 112 + shift;
    const double ar = t[0].warp_sum(ea), ai = t[1].warp_sum(ea), br = t[2].warp_sum(eb), bi = t[3].warp_sum(eb);
    if (lane == 0) {
      h[2 * k] = ar;
      h[2 * k + 1] = ai;
      if (k + 1 < nk) {
        h[2 * k + 2] = br;
        h[2 * k + 3] = bi;
      }
    }
  }
}

// Whether every coefficient is below 2^-36 of |w| (|w|^2 = nn), by exponents, and the
// coefficients times the planes' scale as FP32: value = q1 2^(E - 27). One flag in *ok.
// The FP32 sum is good to about 2^-22 of itself, so below that line it errs by no more
// than 2^-58 sqrt(nk) |w| over the vector; the FP64 form, which rounds w at every
// vector, by about 2^-55 sqrt(nk) |w|.
template <int NT>
__device__ __forceinline__ void plane_coefs(const double* h, const int* qe, int nk, double nn, float2* hf, int* ok) {
  if (threadIdx.x == 0) *ok = 1;
  __syncthreads();
  const int en = (int)(abs_high_word(nn) >> 20) - 1023;
  bool small = true;
  for (int k = threadIdx.x; k < nk; k += NT) {
    const int eh = (int)(max(abs_high_word(h[2 * k]), abs_high_word(h[2 * k + 1])) >> 20) - 1023;
    small = small && 2 * (eh + 2) <= en - 72;
    const int e = qe[k] - 27;
    const float sc = e < -126 ? 0.0f : __uint_as_float((unsigned)(e + 127) << 23);
    hf[k] = make_float2(f64_lead_f32(h[2 * k]) * sc, f64_lead_f32(h[2 * k + 1]) * sc);
  }
  if (!small) atomicExch(ok, 0);
  __syncthreads();
}

// w -= sum_k h_k V_k, the sum in FP32 from the leading planes; this thread's partial |w|^2.
template <int NT>
__device__ __forceinline__ double cgs_update_q(const int* __restrict__ q1, int64_t NP, int nk, const float2* hf,
                                               double* w, int64_t N) {
  double nn = 0.0;
  for (int64_t i = 4 * threadIdx.x; i < N; i += 4 * NT) {
    float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = 0; k < nk; k++) {
      const int4 v = __ldcg(reinterpret_cast<const int4*>(q1 + k * NP + i));
      const float v0 = (float)v.x, v1 = (float)v.y, v2 = (float)v.z, v3 = (float)v.w;
      const float2 c = hf[k];
      d[0] = fmaf(c.x, v0, fmaf(-c.y, v1, d[0]));
      d[1] = fmaf(c.x, v1, fmaf(c.y, v0, d[1]));
      d[2] = fmaf(c.x, v2, fmaf(-c.y, v3, d[2]));
      d[3] = fmaf(c.x, v3, fmaf(c.y, v2, d[3]));
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (i + q < N) {
        const double a = w[i + q] - (double)d[q];
        w[i + q] = a;
        nn += a * a;
      }
  }
  return nn;
}

// Write v (FP64, double i of the vector) into the SpMV input area: FP32 pairs or FP64 (see bspmv).
template <bool CPLX>
__device__ __forceinline__ void stage_x(void* x, int64_t i, double v, bool f32) {
  if (f32) {
    const float2 p = split_f64(v);
    if (CPLX) {
      float* f = reinterpret_cast<float*>(x) + 4 * (i >> 1) + (i & 1);
      f[0] = p.x;
      f[2] = p.y;
    } else {
      reinterpret_cast<float2*>(x)[i] = p;
    }
  } else {
    reinterpret_cast<double*>(x)[i] = v;
  }
}

// u - 1/2, u uniform in (0, 1): splitmix64 (Steele, Lea, Flood 2014) of (seed, stream, index).
__device__ __forceinline__ double splitmix_unit(uint64_t seed, uint64_t stream, uint64_t i) {
  uint64_t z = seed * 0x9E3779B97F4A7C15ULL + stream * 0xD1B54A32D192ED03ULL + (i + 1) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  z ^= z >> 31;
  return ((double)(z >> 11) + 0.5) * (1.0 / 9007199254740992.0) - 0.5;
}

template <int NT, int LPR, bool CPLX, bool F32>
__device__ void run_instance(const BInst& I, int lam, uint64_t seed, double bd_tol, int use_planes, double* sm,
                             void* xs_sm) {
  double* red = sm;
  double* hs = red + RED;
  double* h2 = hs + 2 * (lam + 1);
  double* ta = h2 + 2 * (lam + 1);
  double* tb = ta + lam;
  double* ys = tb + lam + 1;
  double* trw = ys + lam;
  double* scal = trw + 6 * lam;
  void* x = I.xsmem ? xs_sm : static_cast<void*>(I.xg);
  const int64_t N = I.dim * (CPLX ? 2 : 1);
  // planes: per vector an exponent (ys is free until the tridiagonal solve, as is trw)
  const bool planes = CPLX && use_planes && I.q1;
  const int64_t NP = (N + 3) / 4 * 4;
  int* qe = reinterpret_cast<int*>(ys);
  float2* hf = reinterpret_cast<float2*>(trw);
  int* ok = reinterpret_cast<int*>(scal + 1);
  int* w1 = planes ? I.q1 + (int64_t)(lam + 1) * NP : nullptr;
  int* w0 = planes ? I.q0 + (int64_t)(lam + 1) * NP : nullptr;

  // start vector: splitmix64 of (seed, instance number, index) - 1/2, normalized
  double nn = 0.0, z0 = 0.0;
  for (int64_t i = threadIdx.x; i < N; i += NT) {
    const double v = splitmix_unit(seed, (uint64_t)I.number, (uint64_t)i);
    I.V[i] = v;
    nn += v * v;
  }
  block_sum2<NT>(nn, z0, red);
  {
    const double inv = 1.0 / sqrt(nn);
    unsigned hw = 0;
    sweep<NT, 4>(
        N, [&](int i) { return I.V[i]; },
        [&](int i, double u) {
          const double v = u * inv;
          I.V[i] = v;
          stage_x<CPLX>(x, i, v, F32);
          hw = max(hw, abs_high_word(v));
        });
    if (planes) {
      const int E = plane_exponent<NT>(hw, red);
      if (threadIdx.x == 0) qe[0] = E;
      write_planes<NT>(I.V, N, NP, E, I.q1, I.q0);
    }
  }
  if (threadIdx.x == 0) I.ab[lam] = 0.0;  // beta[0]
  __syncthreads();

  int m = lam, passes2 = 0;
  for (int j = 0; j < lam; j++) {
    bspmv<NT, LPR, CPLX, F32>(I, x, I.w, false);
    __syncthreads();
    double n0 = 0.0, z = 0.0;
    if (F32) {
      sweep<NT, 4>(
          N, [&](int i) { return reinterpret_cast<const float2*>(I.w)[i]; },
          [&](int i, float2 pr) {
            const double v = (double)pr.x + (double)pr.y;
            I.w[i] = v;
            n0 += v * v;
          });
      __syncthreads();
    } else {
      for (int64_t i = threadIdx.x; i < N; i += NT) n0 += I.w[i] * I.w[i];
    }
    // three-term step: remove the components along v_{j-1} and v_j
    const int k0 = j > 0 ? j - 1 : 0, nl = j - k0 + 1;
    cgs_dots<NT, CPLX>(I.V + (int64_t)k0 * N, N, nl, I.w, h2);
    block_sum2<NT>(n0, z, red);  // also orders the dots before the update
    double nloc = cgs_update<NT, CPLX>(I.V + (int64_t)k0 * N, N, nl, h2, I.w);
    z = 0.0;
    block_sum2<NT>(nloc, z, red);
    // full classical Gram-Schmidt pass against V_0..V_j
    double n1;
    if (planes) {
      unsigned hw = 0;
      sweep<NT, 4>(
          N, [&](int i) { return I.w[i]; }, [&](int, double v) { hw = max(hw, abs_high_word(v)); });
      const int we = plane_exponent<NT>(hw, red);
      write_planes<NT>(I.w, N, NP, we, w1, w0);
      __syncthreads();
      cgs_dots_q<NT>(I.q1, I.q0, NP, qe, j + 1, w1, w0, we, hs);
      __syncthreads();
      plane_coefs<NT>(hs, qe, j + 1, nloc, hf, ok);
      n1 = *ok ? cgs_update_q<NT>(I.q1, NP, j + 1, hf, I.w, N) : cgs_update<NT, CPLX>(I.V, N, j + 1, hs, I.w);
    } else {
      cgs_dots<NT, CPLX>(I.V, N, j + 1, I.w, hs);
      __syncthreads();
      n1 = cgs_update<NT, CPLX>(I.V, N, j + 1, hs, I.w);
    }
    z = 0.0;
    block_sum2<NT>(n1, z, red);
    for (int t = threadIdx.x; t < 2 * nl; t += NT) hs[2 * k0 + t] += h2[t];
    __syncthreads();
    if (n1 < 0.5 * nloc) {
      // the norm fell below 1/sqrt(2) of its value after the three-term step: repeat the pass
      passes2++;
      cgs_dots<NT, CPLX>(I.V, N, j + 1, I.w, h2);
      __syncthreads();
      n1 = cgs_update<NT, CPLX>(I.V, N, j + 1, h2, I.w);
      z = 0.0;
      block_sum2<NT>(n1, z, red);
      for (int t = threadIdx.x; t < 2 * (j + 1); t += NT) hs[t] += h2[t];
      __syncthreads();
    }
    const double alpha = hs[2 * j];
    const double beta = sqrt(n1);
    const double bprev = I.ab[lam + j];
    __syncthreads();
    if (threadIdx.x == 0) {
      I.ab[j] = alpha;
      I.ab[lam + j + 1] = beta;
    }
    const double scale = fabs(alpha) + bprev;
    if (!(beta > bd_tol * (scale > 0 ? scale : 1.0))) {
      m = j + 1;  // invariant subspace: T is exact
      break;
    }
    if (j + 1 == lam) break;
    const double inv = 1.0 / beta;
    double* vn = I.V + (int64_t)(j + 1) * N;
    unsigned hw = 0;
    sweep<NT, 4>(
        N, [&](int i) { return I.w[i]; },
        [&](int i, double u) {
          const double v = u * inv;
          vn[i] = v;
          stage_x<CPLX>(x, i, v, F32);
          hw = max(hw, abs_high_word(v));
        });
    if (planes) {
      const int E = plane_exponent<NT>(hw, red);
      if (threadIdx.x == 0) qe[j + 1] = E;
      write_planes<NT>(vn, N, NP, E, I.q1 + (int64_t)(j + 1) * NP, I.q0 + (int64_t)(j + 1) * NP);
    }
    __syncthreads();
  }
  __syncthreads();

  // lowest eigenpair of the m x m tridiagonal
  for (int i = threadIdx.x; i < m; i += NT) {
    ta[i] = I.ab[i];
    tb[i] = I.ab[lam + i];
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    double lo = 0.0, hi = 0.0, pm = 0.0;
    if (lane == 0) gersh(ta, tb, m, &lo, &hi, &pm);
    lo = __shfl_sync(0xffffffffu, lo, 0);
    hi = __shfl_sync(0xffffffffu, hi, 0);
    pm = __shfl_sync(0xffffffffu, pm, 0);
    for (int it = 0; it < 40; it++) {
      const double xv = lo + (hi - lo) * (lane + 1) / 33.0;
      const int c = sturm_count(ta, tb, m, xv, pm);
      const unsigned bal = __ballot_sync(0xffffffffu, c >= 1);
      const int first = bal ? __ffs(bal) - 1 : 32;
      const double nlo = first == 0 ? lo : lo + (hi - lo) * first / 33.0;
      const double nhi = first == 32 ? hi : lo + (hi - lo) * (first + 1) / 33.0;
      lo = nlo;
      hi = nhi;
      if (hi - lo <= 2 * DBL_EPSILON * fmax(fabs(lo), fabs(hi))) break;
    }
    if (lane == 0) {
      scal[0] = 0.5 * (lo + hi);
      tri_inverse_iteration(ta, tb, m, scal[0], ys, trw);
    }
  }
  __syncthreads();
  const double theta = scal[0];
  // ground state psi = sum_k y_k V_k, normalized
  nn = 0.0;
  for (int64_t i = threadIdx.x; i < N; i += NT) {
    double acc = 0.0;
    for (int k = 0; k < m; k++) acc += ys[k] * I.V[(int64_t)k * N + i];
    I.psi[i] = acc;
    nn += acc * acc;
  }
  z0 = 0.0;
  block_sum2<NT>(nn, z0, red);
  {
    const double inv = 1.0 / sqrt(nn);
    for (int64_t i = threadIdx.x; i < N; i += NT) {
      const double v = I.psi[i] * inv;
      I.psi[i] = v;
      if (!F32) stage_x<CPLX>(x, i, v, false);
    }
  }
  __syncthreads();
  double energy = theta;
  if (!F32) {
    // Rayleigh quotient with the stored FP64 CSR
    double d = bspmv<NT, LPR, CPLX, false>(I, x, nullptr, true), zz = 0.0;
    block_sum2<NT>(d, zz, red);
    energy = d;
  }
  if (threadIdx.x == 0) {
    const double bm = I.ab[lam + m];
    I.res[0] = energy;
    I.res[1] = theta;
    I.res[2] = fabs(bm * ys[m - 1]);
    I.res[3] = m;
    I.res[4] = passes2;
  }
  __syncthreads();
}

template <int NT, int LPR>
__global__ void __launch_bounds__(NT) k_batch_lanczos(const BInst* __restrict__ insts, const int* __restrict__ order,
                                                      int n, int lam, uint64_t seed, double bd_tol, int use_planes,
                                                      int* counter) {
  extern __shared__ __align__(16) double bsm[];
  void* xs_sm = bsm + batch_fixed_doubles(lam);
  __shared__ int s_idx;
  __shared__ BInst I;  // (its pointers would take thirty registers of every thread)
  for (;;) {
    if (threadIdx.x == 0) {
      s_idx = atomicAdd(counter, 1);
      if (s_idx < n) I = insts[order[s_idx]];
    }
    __syncthreads();
    if (s_idx >= n) break;
    if (I.cplx) {
      if (I.fp32) run_instance<NT, LPR, true, true>(I, lam, seed, bd_tol, use_planes, bsm, xs_sm);
      else run_instance<NT, LPR, true, false>(I, lam, seed, bd_tol, use_planes, bsm, xs_sm);
    } else {
      if (I.fp32) run_instance<NT, LPR, false, true>(I, lam, seed, bd_tol, use_planes, bsm, xs_sm);
      else run_instance<NT, LPR, false, false>(I, lam, seed, bd_tol, use_planes, bsm, xs_sm);
    }
    __syncthreads();  // I and s_idx are written again
  }
}

// res[i][0] = sum of the Rayleigh-quotient block partials of instance i (real parts).
__global__ void k_rq_reduce(const double* __restrict__ part, const int64_t* __restrict__ off,
                            const int* __restrict__ cnt, int n, double* const* res) {
  const int i = blockIdx.x;
  if (i >= n) return;
  __shared__ double red[8];
  double s = 0.0;
  for (int b = threadIdx.x; b < cnt[i]; b += blockDim.x) s += part[2 * (off[i] + b)];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
    res[i][0] = t;
  }
}

// The instances' fixed-point dots of one vector w against nk others into h (blqh_debug_dots)
// or, with hf, their correction of w by given coefficients h (blqh_debug_batch_update).
constexpr int DEBUG_NT = 256;
__global__ void __launch_bounds__(DEBUG_NT) k_debug_pass(const double* V, double* w, int64_t N, int nk, int* q1,
                                                         int* q0, int* qe, double* h, float2* hf) {
  __shared__ double red[RED];
  const int64_t NP = (N + 3) / 4 * 4;
  for (int k = 0; k <= nk; k++) {
    const double* x = k < nk ? V + k * N : w;
    unsigned hw = 0;
    for (int64_t i = threadIdx.x; i < N; i += DEBUG_NT) hw = max(hw, abs_high_word(x[i]));
    const int E = plane_exponent<DEBUG_NT>(hw, red);
    if (threadIdx.x == 0) qe[k] = E;
    write_planes<DEBUG_NT>(x, N, NP, E, q1 + k * NP, q0 + k * NP);
    __syncthreads();
  }
  if (!hf) {
    cgs_dots_q<DEBUG_NT>(q1, q0, NP, qe, nk, q1 + nk * NP, q0 + nk * NP, qe[nk], h);
    return;
  }
  __shared__ int ok;
  double nn = 0.0, z = 0.0;
  for (int64_t i = threadIdx.x; i < N; i += DEBUG_NT) nn += w[i] * w[i];
  block_sum2<DEBUG_NT>(nn, z, red);
  plane_coefs<DEBUG_NT>(h, qe, nk, nn, hf, &ok);
  if (ok) cgs_update_q<DEBUG_NT>(q1, NP, nk, hf, w, N);
  else cgs_update<DEBUG_NT, true>(V, N, nk, h, w);
}

using KFn = void (*)(const BInst*, const int*, int, int, uint64_t, double, int, int*);
KFn batch_kernel(int threads, int lpr) {
#define BLQH_K(T, L) \
  if (threads == T && lpr == L) return k_batch_lanczos<T, L>;
  BLQH_K(256, 4) BLQH_K(256, 8) BLQH_K(256, 16) BLQH_K(256, 32)
  BLQH_K(512, 4) BLQH_K(512, 8) BLQH_K(512, 16) BLQH_K(512, 32)
#undef BLQH_K
  return nullptr;
}

}  // namespace

// ---------------------------------------------------------------------------
struct blqh_batch {
  blqh_ctx* ctx = nullptr;
  blqh_batch_opts o{};
  int n = 0;
  std::vector<blqh_instance> inst;
  std::vector<blqh_basis*> bases;
  std::vector<int> bidx;             // instance -> basis
  std::vector<blqh_csr*> csr;        // null when the sector is empty
  std::vector<RqPlan*> rq;           // mixed precision finisher plans
  std::vector<int64_t> N;            // doubles per vector
  std::vector<size_t> pool_off;      // doubles from the pool start
  double* pool = nullptr;
  int* qpool = nullptr;              // fixed-point planes of the complex instances (of as many as there is room for)
  double* d_resall = nullptr;        // [n][5] results
  BInst* d_inst = nullptr;
  int* d_order = nullptr;
  int* d_counter = nullptr;
  int nrun = 0;                      // instances with dim > 0
  double* d_part = nullptr;          // Rayleigh partials
  int64_t* d_off = nullptr;
  int* d_cnt = nullptr;
  double** d_res = nullptr;
  int nrq = 0;
  int threads = 512, lpr = 16, bps = 1, smem = 0, grid = 0;
  int64_t x_cap = 0;                 // bytes of the shared x area (set_shape may grow it for complex instances)
  int64_t max_n = 0;                 // longest vector
  int fixed = 0, smem_max = 0;       // bytes of the other shared memory; of what a block may have
  std::vector<BInst> hinst;          // the instances that run, as in d_inst
  double mean_row = 0, mean_dim = 0; // over the running instances (tuning class)
  KFn kern = nullptr;
  cudaGraphExec_t gexec = nullptr;
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};  // before the Lanczos launch, after it, after the finisher
  bool solved = false;
  Lay layout(int i) const {
    const bool cplx = csr[i]->is_complex;
    // (the x area may grow after the tuning, so complex instances keep a global one)
    return instance_layout(N[i], o.lambda, !cplx && N[i] * 8 <= x_cap);
  }
};

namespace {

void batch_free(blqh_batch* b) {
  if (!b) return;
  if (b->gexec) cudaGraphExecDestroy(b->gexec);
  for (auto e : b->ev)
    if (e) cudaEventDestroy(e);
  for (auto* p : b->rq)
    if (p) rq_plan_destroy(p);
  for (auto* m : b->csr) free_csr(m);
  for (auto* s : b->bases) blqh_basis_destroy(s);
  dev_free(b->pool);
  dev_free(b->qpool);
  dev_free(b->d_resall);
  dev_free(b->d_inst);
  dev_free(b->d_order);
  dev_free(b->d_counter);
  dev_free(b->d_part);
  dev_free(b->d_off);
  dev_free(b->d_cnt);
  dev_free(b->d_res);
  delete b;
}

int lpr_for(double mean_row) {
  if (mean_row >= 96) return 32;
  if (mean_row >= 40) return 16;
  if (mean_row >= 12) return 8;
  return 4;
}

// Kernel, shared memory and occupancy for a (threads, lanes per row) shape.
void configure_shape(blqh_batch* b, int threads, int lpr) {
  blqh_ctx* ctx = b->ctx;
  b->threads = threads;
  b->lpr = lpr;
  b->kern = batch_kernel(threads, lpr);
  if (!b->kern) {
    set_error(ctx, BLQH_ERR_ARG, "blqh_batch_create: threads 256 or 512, lanes_per_row 4, 8, 16 or 32");
    throw BlqhError{BLQH_ERR_ARG, "shape"};
  }
  BLQH_TRY_CUDA(ctx, smem_attr_at_least(b->kern, b->smem));
  int bps = 0;
  BLQH_TRY_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, b->kern, b->threads, b->smem));
  b->bps = std::max(1, bps);
  b->grid = std::max(1, std::min(b->nrun, ctx->num_sms * b->bps));
}

// A shape with its x area. Where one block per SM is all there is (by its registers and
// shared memory, or by the number of instances), the area takes what shared memory is
// left, so that the gathers of larger complex instances stay in it.
void set_shape(blqh_batch* b, int threads, int lpr) {
  blqh_ctx* ctx = b->ctx;
  int64_t cap = b->x_cap;
  b->smem = b->fixed + (int)((cap + 15) / 16 * 16);
  configure_shape(b, threads, lpr);
  if (b->bps == 1 || b->nrun <= ctx->num_sms) {
    cudaFuncAttributes fa;  // the kernel's own static shared memory counts against the limit
    BLQH_TRY_CUDA(ctx, cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(b->kern)));
    const int64_t room = (b->smem_max - b->fixed - (int64_t)fa.sharedSizeBytes) / 16 * 16;
    const int64_t grown = std::min<int64_t>((b->max_n * 8 + 15) / 16 * 16, room);
    if (grown > cap) {
      cap = grown;
      b->smem = b->fixed + (int)cap;
      configure_shape(b, threads, lpr);
    }
  }
  bool changed = false;
  for (BInst& I : b->hinst) {
    const int fits = I.dim * 16 <= cap;
    if (!I.cplx || I.xsmem == fits) continue;
    I.xsmem = fits;
    changed = true;
  }
  if (changed)
    BLQH_TRY_CUDA(ctx, cudaMemcpy(b->d_inst, b->hinst.data(), b->hinst.size() * sizeof(BInst), cudaMemcpyHostToDevice));
}

// K10 for the batch: each candidate shape runs one round of the most
// expensive instances (one per resident block) for a few Lanczos steps on the
// batch's own data, as the solve will run them; the fastest per instance-step wins and
// is cached per class (batches with planes and without are two; v2: the shape's x area
// and the planes are part of what was timed).
void tune_shape(blqh_batch* b) {
  blqh_ctx* ctx = b->ctx;
  int kind = 0;  // 1: complex instances among them, 2: with planes
  for (const BInst& I : b->hinst) kind = std::max(kind, I.cplx ? (I.q1 ? 2 : 1) : 0);
  const std::string key = tune_key("batch|v2", b->o.value_precision, kind, (int64_t)b->mean_dim, b->mean_row,
                                   b->o.lambda);
  int t = 0, l = 0;
  if (!tune_lookup(key, &t, &l)) {
    const int lam_t = std::min(b->o.lambda, 12);
    double best = 1e30;
    for (int th : {256, 512})
      for (int lp : {4, 8, 16, 32}) {
        if (lp == 4 && b->mean_row >= 24) continue;
        set_shape(b, th, lp);
        const int nsub = std::min(b->nrun, ctx->num_sms * b->bps);
        double ms_best = 1e30;
        for (int rep = 0; rep < 2; rep++) {
          BLQH_TRY_CUDA(ctx, cudaMemsetAsync(b->d_counter, 0, sizeof(int), ctx->stream));
          BLQH_TRY_CUDA(ctx, cudaEventRecord(b->ev[0], ctx->stream));
          b->kern<<<std::min(b->grid, nsub), b->threads, b->smem, ctx->stream>>>(b->d_inst, b->d_order, nsub, lam_t,
                                                                                 b->o.seed, 1e-13, 1, b->d_counter);
          BLQH_TRY_CUDA(ctx, cudaGetLastError());
          BLQH_TRY_CUDA(ctx, cudaEventRecord(b->ev[1], ctx->stream));
          BLQH_TRY_CUDA(ctx, cudaEventSynchronize(b->ev[1]));
          float ms = 0;
          BLQH_TRY_CUDA(ctx, cudaEventElapsedTime(&ms, b->ev[0], b->ev[1]));
          ms_best = std::min(ms_best, (double)ms);
        }
        const double per = ms_best / nsub;  // time per instance over the round
        if (per < best) {
          best = per;
          t = th;
          l = lp;
        }
      }
    tune_store(key, t, l, best);
  }
  set_shape(b, t, l);
}

void batch_create_impl(blqh_batch* b) {
  blqh_ctx* ctx = b->ctx;
  const int lam = b->o.lambda;
  // one basis per distinct sector
  std::map<std::tuple<int, int, int, int, int, int, int, int>, int> seen;
  b->bidx.resize(b->n);
  for (int i = 0; i < b->n; i++) {
    const int model = b->inst[i].model;
    const blqh_sector& s = b->inst[i].sector;
    const blqh_sector_spin& ss = b->inst[i].ssector;
    const blqh_sector_mono& ms = b->inst[i].msector;
    const auto key = model == BLQH_MODEL_SPINFUL
                         ? std::make_tuple(1, ss.nphi, ss.nel, ss.nel_up, ss.nel_su, ss.J, ss.K, ss.rep_mode)
                     : model == BLQH_MODEL_MONOLAYER ? std::make_tuple(2, ms.nphi, ms.nel, -1, -1, ms.J, ms.K, ms.rep_mode)
                                                     : std::make_tuple(0, s.nphi, s.nel, s.nel_up, -1, s.J, s.K, s.rep_mode);
    auto it = seen.find(key);
    if (it == seen.end()) {
      blqh_basis* B = nullptr;
      const int rc = model == BLQH_MODEL_SPINFUL     ? blqh_basis_build_spin(ctx, &ss, &B)
                     : model == BLQH_MODEL_MONOLAYER ? blqh_basis_build_mono(ctx, &ms, &B)
                                                     : blqh_basis_build(ctx, &s, &B);
      if (rc != BLQH_OK) throw BlqhError{rc, "basis"};
      it = seen.emplace(key, (int)b->bases.size()).first;
      b->bases.push_back(B);
    }
    b->bidx[i] = it->second;
  }
  // CSR per instance
  b->csr.assign(b->n, nullptr);
  b->N.assign(b->n, 0);
  double nnz_sum = 0, dim_sum = 0;
  for (int i = 0; i < b->n; i++) {
    const blqh_basis* B = b->bases[b->bidx[i]];
    if (B->dim == 0) continue;
    blqh_csr* M = new blqh_csr;
    M->ctx = ctx;
    b->csr[i] = M;
    if (b->inst[i].model == BLQH_MODEL_SPINFUL) {
      spin_hamil_build_impl(ctx, B, b->inst[i].sparams, M);
    } else if (b->inst[i].model == BLQH_MODEL_MONOLAYER) {
      mono_hamil_build_impl(ctx, B, b->inst[i].mparams, M);
    } else {
      hamil_build_impl(ctx, B, b->inst[i].params, b->o.value_precision, M);
    }
    b->N[i] = M->dim * (M->is_complex ? 2 : 1);
    nnz_sum += (double)M->nnz;
    dim_sum += (double)M->dim;
    b->max_n = std::max(b->max_n, b->N[i]);
  }
  // shared memory: the fixed part plus an x area for the instances that fit in it
  cudaDeviceGetAttribute(&b->smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
  b->fixed = batch_fixed_doubles(lam) * 8;
  const int64_t x_cap = std::min<int64_t>(b->max_n * 8, (int64_t)std::max(0, 96 * 1024 - b->fixed));
  b->x_cap = x_cap;
  b->smem = b->fixed + (int)((x_cap + 15) / 16 * 16);
  if (b->smem > b->smem_max) {
    set_error(ctx, BLQH_ERR_UNSUPPORTED, "blqh_batch_create: lambda too large for shared memory");
    throw BlqhError{BLQH_ERR_UNSUPPORTED, "smem"};
  }
  for (auto& e : b->ev) BLQH_TRY_CUDA(ctx, cudaEventCreate(&e));
  // shape: threads and lanes per row (given, tuned, or the defaults)
  b->mean_row = dim_sum > 0 ? nnz_sum / dim_sum : 0;
  b->mean_dim = b->n ? dim_sum / std::max(1, (int)std::count_if(b->csr.begin(), b->csr.end(), [](blqh_csr* m) {
    return m != nullptr;
  })) : 0;
  configure_shape(b, b->o.threads ? b->o.threads : 256,
                  b->o.lanes_per_row ? b->o.lanes_per_row : lpr_for(b->mean_row));
  // device storage per instance (instance_layout)
  b->pool_off.assign(b->n, 0);
  size_t total = 0;
  for (int i = 0; i < b->n; i++) {
    if (!b->csr[i]) continue;
    b->pool_off[i] = total;
    total += b->layout(i).total;
  }
  b->pool = dalloc<double>(ctx, total + 32);
  // planes (as much again) for the first complex instances that half of the free memory
  // holds; the others take the FP64 pass
  std::vector<size_t> plane_at(b->n, SIZE_MAX);
  size_t ints = 0;
  const size_t room = optional_bytes(ctx) / sizeof(int);
  for (int i = 0; i < b->n; i++) {
    const size_t need = b->csr[i] && b->csr[i]->is_complex ? 2 * plane_ints(b->N[i], lam) : 0;
    if (!need || ints + need > room) continue;
    plane_at[i] = ints;
    ints += need;
  }
  if (ints) try {
      b->qpool = dalloc<int>(ctx, ints);
    } catch (const BlqhError& e) {
      if (e.code != BLQH_ERR_NOMEM) throw;
      ctx->last_error.clear();
    }
  b->d_resall = dalloc<double>(ctx, 5 * (size_t)std::max(1, b->n));  // every instance's results, read back at once
  std::vector<BInst>& hi = b->hinst;
  std::vector<double> cost;
  std::vector<double*> res_ptr;
  for (int i = 0; i < b->n; i++) {
    if (!b->csr[i]) continue;
    const blqh_csr* M = b->csr[i];
    BInst I{};
    I.rp = M->d_row_ptr;
    I.col = M->d_col;
    I.val = M->d_val;
    I.dim = M->dim;
    I.cplx = M->is_complex;
    I.fp32 = M->precision == BLQH_VAL_FP32;
    const int64_t Ni = b->N[i];
    I.xsmem = Ni * 8 <= x_cap;
    I.number = i;
    double* p = b->pool + b->pool_off[i];
    const Lay L = b->layout(i);
    I.V = p + L.V;
    I.w = p + L.w;
    I.psi = p + L.psi;
    I.ab = p + L.ab;
    I.res = b->d_resall + 5 * (size_t)i;
    I.xg = I.xsmem && !I.cplx ? nullptr : p + L.xg;
    if (b->qpool && plane_at[i] != SIZE_MAX) {
      I.q1 = b->qpool + plane_at[i];
      I.q0 = I.q1 + plane_ints(Ni, lam);
    }
    hi.push_back(I);
    // cost: SpMV bytes and reorthogonalization work over lam steps
    cost.push_back((double)lam * ((double)M->nnz * (I.fp32 ? 8.0 : 12.0) * (I.cplx ? 1.5 : 1.0) +
                                  0.5 * lam * (double)Ni * 16.0));
  }
  b->nrun = (int)hi.size();
  std::vector<int> order(b->nrun);
  for (int k = 0; k < b->nrun; k++) order[k] = k;
  std::stable_sort(order.begin(), order.end(), [&](int a, int c) { return cost[a] > cost[c]; });
  b->d_inst = dalloc<BInst>(ctx, std::max(1, b->nrun));
  b->d_order = dalloc<int>(ctx, std::max(1, b->nrun));
  b->d_counter = dalloc<int>(ctx, 1);
  if (b->nrun) {
    BLQH_TRY_CUDA(ctx, cudaMemcpy(b->d_inst, hi.data(), hi.size() * sizeof(BInst), cudaMemcpyHostToDevice));
    BLQH_TRY_CUDA(ctx, cudaMemcpy(b->d_order, order.data(), order.size() * sizeof(int), cudaMemcpyHostToDevice));
  }
  b->grid = std::max(1, std::min(b->nrun, ctx->num_sms * b->bps));
  if (b->nrun) {
    if (b->o.threads == 0 && b->o.lanes_per_row == 0 && tune_enabled()) tune_shape(b);
    else set_shape(b, b->threads, b->lpr);
  }
  // mixed precision: one regenerated Rayleigh quotient per instance
  b->rq.assign(b->n, nullptr);
  if (b->o.value_precision == BLQH_VAL_FP32) {
    std::vector<int64_t> off;
    std::vector<int> cnt;
    int64_t tot = 0;
    int k = 0;  // position among the running instances
    for (int i = 0; i < b->n; i++) {
      if (!b->csr[i]) continue;
      const int kk = k++;
      if (b->csr[i]->precision != BLQH_VAL_FP32) continue;  // spinful: FP64 values, finished in the kernel
      res_ptr.push_back(hi[kk].res);
      b->rq[i] = rq_plan_create(ctx, b->bases[b->bidx[i]], b->inst[i].params);
      off.push_back(tot);
      cnt.push_back(rq_plan_grid(b->rq[i]));
      tot += rq_plan_grid(b->rq[i]);
    }
    b->nrq = (int)off.size();
    b->d_part = dalloc<double>(ctx, 2 * std::max<int64_t>(1, tot));
    b->d_off = dalloc<int64_t>(ctx, std::max(1, b->nrq));
    b->d_cnt = dalloc<int>(ctx, std::max(1, b->nrq));
    b->d_res = dalloc<double*>(ctx, std::max(1, b->nrq));
    if (b->nrq) {
      BLQH_TRY_CUDA(ctx, cudaMemcpy(b->d_off, off.data(), off.size() * 8, cudaMemcpyHostToDevice));
      // (res_ptr lists the instances with a plan, in plan order)
      BLQH_TRY_CUDA(ctx, cudaMemcpy(b->d_cnt, cnt.data(), cnt.size() * 4, cudaMemcpyHostToDevice));
      BLQH_TRY_CUDA(ctx, cudaMemcpy(b->d_res, res_ptr.data(), res_ptr.size() * sizeof(double*),
                                    cudaMemcpyHostToDevice));
    }
  }
  BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
}

// Timing event on the context stream; inside a stream capture it must be an
// external record node (a plain record there only orders work).
void record_ev(blqh_ctx* ctx, cudaEvent_t e) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  BLQH_TRY_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &st));
  if (st == cudaStreamCaptureStatusActive)
    BLQH_TRY_CUDA(ctx, cudaEventRecordWithFlags(e, ctx->stream, cudaEventRecordExternal));
  else
    BLQH_TRY_CUDA(ctx, cudaEventRecord(e, ctx->stream));
}

// Every launch of one solve, in stream order.
void batch_enqueue(blqh_batch* b) {
  blqh_ctx* ctx = b->ctx;
  if (!b->nrun) return;
  BLQH_TRY_CUDA(ctx, cudaMemsetAsync(b->d_counter, 0, sizeof(int), ctx->stream));
  record_ev(ctx, b->ev[0]);
  b->kern<<<b->grid, b->threads, b->smem, ctx->stream>>>(b->d_inst, b->d_order, b->nrun, b->o.lambda, b->o.seed,
                                                         1e-13, 1, b->d_counter);
  BLQH_TRY_CUDA(ctx, cudaGetLastError());
  record_ev(ctx, b->ev[1]);
  count_launch(ctx, TM_SPMV);
  if (b->o.value_precision == BLQH_VAL_FP32) {
    int64_t off = 0;
    for (int i = 0; i < b->n; i++) {
      if (!b->rq[i]) continue;
      const double* psi = b->pool + b->pool_off[i] + b->layout(i).psi;
      rq_plan_launch(ctx, b->rq[i], psi, b->d_part + 2 * off);
      off += rq_plan_grid(b->rq[i]);
    }
    k_rq_reduce<<<b->nrq, 256, 0, ctx->stream>>>(b->d_part, b->d_off, b->d_cnt, b->nrq, b->d_res);
    BLQH_TRY_CUDA(ctx, cudaGetLastError());
    count_launch(ctx, TM_MISC);
  }
  record_ev(ctx, b->ev[2]);
}

void batch_solve_impl(blqh_batch* b) {
  blqh_ctx* ctx = b->ctx;
  if (b->o.use_graph && b->nrun) {
    if (!b->gexec) {
      const bool timing = ctx->timing;
      ctx->timing = false;  // no timer events inside the capture
      cudaGraph_t g = nullptr;
      BLQH_TRY_CUDA(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed));
      try {
        batch_enqueue(b);
      } catch (...) {
        cudaStreamEndCapture(ctx->stream, &g);
        if (g) cudaGraphDestroy(g);
        ctx->timing = timing;
        throw;
      }
      BLQH_TRY_CUDA(ctx, cudaStreamEndCapture(ctx->stream, &g));
      ctx->timing = timing;
      const cudaError_t e = cudaGraphInstantiate(&b->gexec, g, 0);
      cudaGraphDestroy(g);
      BLQH_TRY_CUDA(ctx, e);
    }
    BLQH_TRY_CUDA(ctx, cudaGraphLaunch(b->gexec, ctx->stream));
  } else {
    TimerScope ts(ctx, TM_SPMV);
    batch_enqueue(b);
  }
  BLQH_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (auto* p : b->rq)
    if (p) {
      const int rc = rq_plan_check(ctx, p);
      if (rc) throw BlqhError{rc, "rq"};
    }
  b->solved = true;
}

}  // namespace

// Complex vectors of N doubles, device pointers (see blqh_debug_dots and, with update, blqh_debug_batch_update).
void debug_batch_pass(blqh_ctx* ctx, const double* V, double* w, int64_t N, int nk, double* h, bool update) {
  DevBufs G;
  const size_t NP = (size_t)(N + 3) / 4 * 4;
  int* q1 = G.add(dalloc<int>(ctx, NP * (nk + 1)));
  int* q0 = G.add(dalloc<int>(ctx, NP * (nk + 1)));
  int* qe = G.add(dalloc<int>(ctx, nk + 1));
  float2* hf = update ? G.add(dalloc<float2>(ctx, nk)) : nullptr;
  k_debug_pass<<<1, DEBUG_NT, 0, ctx->stream>>>(V, w, N, nk, q1, q0, qe, h, hf);
  BLQH_TRY_CUDA(ctx, cudaGetLastError());
}

extern "C" {

int blqh_batch_create(blqh_ctx* ctx, const blqh_instance* inst, int n, const blqh_batch_opts* o, blqh_batch** out) {
  if (!ctx || !o || !out || n < 0 || (n > 0 && !inst)) return BLQH_ERR_ARG;
  *out = nullptr;
  if (o->lambda < 2 || o->lambda > 1024 ||
      (o->value_precision != BLQH_VAL_FP32 && o->value_precision != BLQH_VAL_FP64)) {
    set_error(ctx, BLQH_ERR_ARG, "blqh_batch_create: lambda in [2, 1024], value_precision FP32 or FP64");
    return BLQH_ERR_ARG;
  }
  for (int i = 0; i < n; i++)
    if (inst[i].model != BLQH_MODEL_SPINLESS && inst[i].model != BLQH_MODEL_SPINFUL &&
        inst[i].model != BLQH_MODEL_MONOLAYER) {
      set_error(ctx, BLQH_ERR_UNSUPPORTED, "blqh_batch_create: unknown model");
      return BLQH_ERR_UNSUPPORTED;
    }
  blqh_batch* b = new blqh_batch;
  b->ctx = ctx;
  b->o = *o;
  b->n = n;
  b->inst.assign(inst, inst + n);
  try {
    cudaSetDevice(ctx->device);
    batch_create_impl(b);
  } catch (const BlqhError& e) {
    batch_free(b);
    return e.code;
  }
  *out = b;
  return BLQH_OK;
}

int blqh_batch_solve(blqh_batch* b) {
  if (!b) return BLQH_ERR_ARG;
  try {
    cudaSetDevice(b->ctx->device);
    batch_solve_impl(b);
  } catch (const BlqhError& e) {
    return e.code;
  }
  return BLQH_OK;
}

int blqh_batch_results(const blqh_batch* b, blqh_batch_result* out) {
  if (!b || !out) return BLQH_ERR_ARG;
  if (!b->solved) {
    set_error(b->ctx, BLQH_ERR_STATE, "blqh_batch_results: call blqh_batch_solve first");
    return BLQH_ERR_STATE;
  }
  std::vector<double> all(5 * (size_t)std::max(1, b->n));
  if (b->nrun &&
      cudaMemcpy(all.data(), b->d_resall, 5 * (size_t)b->n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) {
    set_error(b->ctx, BLQH_ERR_CUDA, "blqh_batch_results: copy failed");
    return BLQH_ERR_CUDA;
  }
  for (int i = 0; i < b->n; i++) {
    blqh_batch_result r{};
    const blqh_csr* M = b->csr[i];
    if (!M) {
      r.energy = r.ritz0 = NAN;
      out[i] = r;
      continue;
    }
    const double* res = all.data() + 5 * (size_t)i;
    r.energy = res[0];
    r.ritz0 = res[1];
    r.resid = res[2];
    r.steps = (int)res[3];
    r.second_passes = (int)res[4];
    r.dim = M->dim;
    r.nnz = M->nnz;
    out[i] = r;
  }
  return BLQH_OK;
}

int blqh_batch_ground_state(const blqh_batch* b, int i, double* psi) {
  if (!b || !psi || i < 0 || i >= b->n) return BLQH_ERR_ARG;
  if (!b->solved || !b->csr[i]) {
    set_error(b->ctx, BLQH_ERR_STATE, "blqh_batch_ground_state: instance not solved (or empty sector)");
    return BLQH_ERR_STATE;
  }
  const double* d = b->pool + b->pool_off[i] + b->layout(i).psi;
  if (cudaMemcpy(psi, d, b->N[i] * 8, cudaMemcpyDeviceToHost) != cudaSuccess) {
    set_error(b->ctx, BLQH_ERR_CUDA, "blqh_batch_ground_state: copy failed");
    return BLQH_ERR_CUDA;
  }
  return BLQH_OK;
}

int blqh_batch_shape(const blqh_batch* b, int* threads, int* lanes_per_row, int* blocks_per_sm) {
  if (!b) return BLQH_ERR_ARG;
  if (threads) *threads = b->threads;
  if (lanes_per_row) *lanes_per_row = b->lpr;
  if (blocks_per_sm) *blocks_per_sm = b->bps;
  return BLQH_OK;
}

int blqh_batch_timing(const blqh_batch* b, double* lanczos_ms, double* finish_ms, int* launches) {
  if (!b) return BLQH_ERR_ARG;
  if (!b->solved || !b->nrun) {
    set_error(b->ctx, BLQH_ERR_STATE, "blqh_batch_timing: no solve has run");
    return BLQH_ERR_STATE;
  }
  float a = 0.f, c = 0.f;
  if (cudaEventElapsedTime(&a, b->ev[0], b->ev[1]) != cudaSuccess ||
      cudaEventElapsedTime(&c, b->ev[1], b->ev[2]) != cudaSuccess) {
    cudaGetLastError();
    set_error(b->ctx, BLQH_ERR_CUDA, "blqh_batch_timing: event timing unavailable");
    return BLQH_ERR_CUDA;
  }
  if (lanczos_ms) *lanczos_ms = a;
  if (finish_ms) *finish_ms = c;
  if (launches) *launches = 1 + (b->o.value_precision == BLQH_VAL_FP32 ? b->nrq + 1 : 0);
  return BLQH_OK;
}

int blqh_batch_destroy(blqh_batch* b) {
  batch_free(b);
  return BLQH_OK;
}

int blqh_batch_run(blqh_ctx* ctx, const blqh_instance* inst, int n, const blqh_batch_opts* o,
                   blqh_batch_result* out) {
  if (!out && n > 0) return BLQH_ERR_ARG;
  blqh_batch* b = nullptr;
  int rc = blqh_batch_create(ctx, inst, n, o, &b);
  if (rc == BLQH_OK) rc = blqh_batch_solve(b);
  if (rc == BLQH_OK) rc = blqh_batch_results(b, out);
  blqh_batch_destroy(b);
  return rc;
}

}  // extern "C"
