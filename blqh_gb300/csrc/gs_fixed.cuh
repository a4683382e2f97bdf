// The Lanczos step after the SpMV for complex sectors: three-term update and one
// classical Gram-Schmidt pass against every stored vector, on fixed-point planes.
// (Real sectors keep a fixed order of operations: gs_ordered.cuh.)
//
// GB300's FP64 pipe issues ~2 lane operations per clock per SM (measured: DFMA
// 1.6, FFMA 118, IMAD.WIDE with 64-bit accumulation 27 lanes per clock per SM),
// so FP64 dots against j stored vectors ran at 35 % of HBM bandwidth with that
// pipe 88 % busy, and double-float dots on the FP32 pipes carry 2^-46. Here every
// Krylov vector is kept a second time as integers: per tile of TILE consecutive
// doubles with 2^E <= max|x| < 2^(E+1),
//   x = q 2^(E-56), |q| <= 2^57, q = q1 2^29 + q0, |q1| <= 2^28, |q0| <= 2^28,
// in two int32 planes Q1, Q0 and one exponent per tile. A dot of two tiles is
// then exact integer arithmetic: four IMAD.WIDE per product into three 64-bit
// sums per lane (32 products per lane: |q1 w1| sums below 2^61, the cross terms
// below 2^62), one 128-bit sum over the warp, one conversion to FP64 per (tile,
// vector); tiles are summed in FP64. What is lost is the operands' rounding at 2^-57
// of the tile's largest entry (an entry below a sixteenth of that keeps fewer than
// FP64's 53 bits), but no product or sum within a tile rounds: error against extended
// precision 0.33 to 0.80 of the FP64 dots', random vectors of 79 to 100,141 complex
// entries (tests/test_fixed_dots.py). The dots read 8 bytes per entry as before.
//
// The pass's correction sum_k h_k V_k (every |h_k| <= 2^-30 |w|, checked per
// step, else FP64) is summed in FP32 from the Q1 plane alone (4 bytes per entry,
// 2^-29 of the tile's maximum) and subtracted from w in FP64.
//
// beta_{j+1}^2 = |w|^2 - sum_k |h_k|^2, exact to FP64's rounding under the same
// bound, so the kernel that subtracts the correction also writes v_{j+1} and its
// planes: w is not stored and read again, and one grid-wide reduction falls away.
//
// A step's kernels after the SpMV: k_alpha (partials of v_j w), k_local (w' = w -
// alpha_j v_j and its planes), k_dots_q, k_update_q. On short sectors (256-entry
// tiles) k_local is left out: every block of the other two takes its own tile of
// w' from w and v_j. Small sectors are bound by the chain of dependent reads, so
// reductions whose partials are few are summed by the kernels that need them, in
// the same order in every block (no arrival counter, no extra round trip); only
// the dots, nk times as many, end in their group's last block. Each kernel is
// launched with programmatic stream serialization: its blocks are placed while the
// previous kernel drains. Results are reproducible.
//
// Measured per step without the SpMV (200 steps, one GB300): 60,096 rows 300 -> 52
// us, 100,141 rows 311 -> 78 us, 647,079 rows (FP32 values) 496 -> 355 us, 16,024
// rows 251 -> 34 us.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

// device scalar block layout (doubles), per Lanczos object
struct Scal {
  double* alpha;  // [mmax]
  double* beta;   // [mmax+1]; beta[0] = 0 internally
  double* h2;     // [2*(mmax+1)] coefficients of the full pass (re, im)
  double* nrm;    // [4]: [2], [3] scratch
  double* ritz;   // [mmax] lowest Ritz value at checks
  int* flags;     // [8]: stop, -, steps, breakdown, a coefficient of the ordered full pass not small,
                  //      the tridiagonal size of the last convergence check's Ritz value
  unsigned* cnt;  // arrival counters of the kernels that end in their last block (zero between launches)
};

enum { CNT_UPDATE = 0, CNT_DOTS = 2 };

// Blocks of the next kernel may be placed from here on; this kernel's reads of
// the previous one's results start after the wait.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Sum over the block (a multiple of 32 threads; red: one double per warp), valid in thread 0.
__device__ __forceinline__ double block_sum_256(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) s += red[i];
  __syncthreads();
  return s;
}

// True in every thread of the last of `nblk` blocks to arrive at *cnt, whose
// partials (written before the call) are then all visible; the counter is back
// at zero afterwards.
__device__ __forceinline__ bool last_block(unsigned* cnt, unsigned nblk) {
  __shared__ bool last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc(cnt, nblk - 1) == nblk - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// FP32 value with the 24 leading significant bits of x (truncated), from its
// bit pattern with integer operations only (GB300's FP64 pipe issues ~2 lane
// operations per clock per SM; this keeps the correction below off it).
// |x| < 2^-126 gives 0; |x| < 2^128 is assumed (Krylov vectors have |x| <= 1).
__device__ __forceinline__ float f64_lead_f32(double x) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const unsigned hw = (unsigned)(bits >> 32), lw = (unsigned)bits;
  const int e = (int)((hw >> 20) & 0x7FFu) - 896;  // FP32 biased exponent
  const unsigned f = (hw & 0x80000000u) | ((unsigned)e << 23) | (__funnelshift_l(lw, hw, 3) & 0x7FFFFFu);
  return e > 0 ? __uint_as_float(f) : 0.0f;
}

// beta_{j+1} = |w| from the final |w|^2, the step count, and the breakdown test
// (one thread).
__device__ __forceinline__ void beta_from(const Scal& S, int j, double nrm2, double breakdown_tol) {
  const double b = sqrt(nrm2);
  S.beta[j + 1] = b;
  S.flags[2] = j + 1;
  const double scale = fabs(S.alpha[j]) + S.beta[j];
  if (!(b > breakdown_tol * (scale > 0 ? scale : 1.0))) {
    S.flags[3] = 1;
    S.flags[0] = 1;
  }
}

// ---------------------------------------------------------------------------
// Fixed point: x = (q1 2^29 + q0) 2^(E-56), rounded to nearest; 2^E <= |x|max of
// the tile. Bit operations only. Denormals count as zero.
__device__ __forceinline__ void quantize(double x, int E, int& q1, int& q0) {
  const long long b = __double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7FF);
  long long m = ((b & 0xFFFFFFFFFFFFFLL) | 0x10000000000000LL) << 4;
  const int sh = E - (ex - 1023);
  if (ex == 0 || sh > 60) m = 0;
  else if (sh > 0) m = (m + (1LL << (sh - 1))) >> sh;
  const long long q = b < 0 ? -m : m;
  q1 = (int)((q + (1LL << 28)) >> 29);
  q0 = (int)(q - ((long long)q1 << 29));
}

// x = (q.x 2^29 + q.y) 2^(xe - 59), |x| <= 2^xe, rounded to nearest (the vector operand
// of the fixed-point SpMV). Larger and non-finite values give zero (the SpMV's FP64
// diagonal term carries them on).
__device__ __forceinline__ int2 fix_scaled(double x, int xe) {
  const long long b = __double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7FF) - 1023;
  long long m = (b & 0xFFFFFFFFFFFFFLL) | 0x10000000000000LL;
  const int sh = ex - xe + 7;  // m 2^(ex - 52) in units of 2^(xe - 59)
  if (sh > 7 || sh < -60) m = 0;
  else if (sh >= 0) m <<= sh;
  else m = (m + (1LL << (-sh - 1))) >> -sh;
  const long long q = b < 0 ? -m : m;
  const int hi = (int)((q + (1LL << 28)) >> 29);
  return make_int2(hi, (int)(q - ((long long)hi << 29)));
}

// Largest value over the block, in every thread.
__device__ __forceinline__ unsigned block_max(unsigned hw, unsigned* red) {
  hw = __reduce_max_sync(0xffffffffu, hw);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = hw;
  __syncthreads();
  unsigned m = 0;
  for (int i = 0; i < (int)(blockDim.x >> 5); i++) m = max(m, red[i]);
  return m;
}

// High word of |x|, and the exponent E of the value it is the high word of (zero and
// denormals: -1023).
__device__ __forceinline__ unsigned abs_high_word(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }
__device__ __forceinline__ int word_exponent(unsigned hw) { return (int)(hw >> 20) - 1023; }

// Exponent E of the largest |x| over the block, from each thread's largest high word.
__device__ __forceinline__ int block_exponent(unsigned hw, unsigned* red) { return word_exponent(block_max(hw, red)); }

// xe of a normalized vector v = (w - c) inv for fix_scaled, 2^E <= max |w| < 2^(E+1),
// |c| <= sqrt(cc): a power of two above |v| (at most 4 times the largest entry for
// negligible c), and no more than 2^0. Integers only, one lane's FP64 would hold the block up.
__device__ __forceinline__ int scaled_exponent(int E, double cc, double inv) {
  const int C = (word_exponent(abs_high_word(cc)) + 2) >> 1;  // sqrt(cc) < 2^C
  const int sum = C < E - 20 ? E + 1 : max(E + 1, C) + 1;     // |w| + |c| < 2^sum (1 + 2^-20)
  return min(sum + word_exponent(abs_high_word(inv) + 4) + 1, 0);
}

// Sum of a pair over the warp, in every lane. (One warp sums what a block needs: an
// FP64 instruction takes the SM's FP64 pipe 16 clocks, so the same sum spread over
// 32 warps costs microseconds.)
__device__ __forceinline__ double2 warp_sum(double2 s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
    s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
  }
  return s;
}
__device__ __forceinline__ double warp_sum(double s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
// Sums of n partials by one warp, in every lane.
__device__ __forceinline__ double2 sum_partials(const double2* p, int n) {
  double2 s = make_double2(0.0, 0.0);
  for (int t = threadIdx.x & 31; t < n; t += 32) {
    const double2 v = __ldcg(p + t);
    s.x += v.x;
    s.y += v.y;
  }
  return warp_sum(s);
}
__device__ __forceinline__ double sum_partials(const double* p, int n) {
  double s = 0.0;
  for (int t = threadIdx.x & 31; t < n; t += 32) s += __ldcg(p + t);
  return warp_sum(s);
}

// Block partials (re, im) of h_j = conj(V_j) w, w after the SpMV.
static __global__ void __launch_bounds__(256) k_alpha(const double* vj, const double* w, int64_t dim, double2* part, Scal S) {
  pdl_begin();
  __shared__ double red[8];
  double sr = 0, si = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += stride) {
    const double2 a = reinterpret_cast<const double2*>(vj)[i], b = reinterpret_cast<const double2*>(w)[i];
    sr += a.x * b.x + a.y * b.y;
    si += a.x * b.y - a.y * b.x;
  }
  if (S.flags[0]) return;
  sr = block_sum_256(sr, red);
  si = block_sum_256(si, red);
  if (threadIdx.x == 0) part[blockIdx.x] = make_double2(sr, si);
}

// w' = w - h v for one complex entry.
__device__ __forceinline__ double2 three_term(double2 w, double2 v, double2 h) {
  return make_double2(w.x - (h.x * v.x - h.y * v.y), w.y - (h.x * v.y + h.y * v.x));
}

// Three-term step: w -= h_j V_j (the SpMV removed beta_j v_{j-1}), partials of
// |w|^2 per tile, and w's fixed-point planes for the full pass. One block of TILE / 4
// threads per tile.
template <int TILE>
__global__ void __launch_bounds__(TILE / 4) k_local(const double* vj, double* w, int64_t n, const double2* apart,
                                                    int na, int* w1, int* w0, int* we, double* part, Scal S, int j) {
  pdl_begin();
  constexpr int T = TILE / 4;
  __shared__ double red[T / 32];
  __shared__ unsigned ured[T / 32];
  __shared__ double2 s_h;
  const int64_t e0 = (int64_t)blockIdx.x * TILE;
  const int stop = S.flags[0];
  double a[4], v[4];
#pragma unroll
  for (int q = 0; q < 4; q += 2) {
    const int64_t i = e0 + 2 * ((q >> 1) * T + threadIdx.x);
    const bool in = i < n;
    const double2 x = in ? *reinterpret_cast<const double2*>(w + i) : make_double2(0.0, 0.0);
    const double2 y = in ? *reinterpret_cast<const double2*>(vj + i) : make_double2(0.0, 0.0);
    a[q] = x.x;
    a[q + 1] = x.y;
    v[q] = y.x;
    v[q + 1] = y.y;
  }
  if (stop) return;
  if (threadIdx.x < 32) {
    const double2 t = sum_partials(apart, na);
    if (threadIdx.x == 0) {
      s_h = t;
      if (blockIdx.x == 0) S.alpha[j] = t.x;
    }
  }
  __syncthreads();
  const double2 h = s_h;
  double nn = 0;
  unsigned hw = 0;
#pragma unroll
  for (int q = 0; q < 4; q += 2) {
    const int64_t i = e0 + 2 * ((q >> 1) * T + threadIdx.x);
    const double2 x = three_term(make_double2(a[q], a[q + 1]), make_double2(v[q], v[q + 1]), h);
    if (i < n) *reinterpret_cast<double2*>(w + i) = x;
    a[q] = x.x;
    a[q + 1] = x.y;
    nn += x.x * x.x + x.y * x.y;
    hw = max(hw, max(abs_high_word(x.x), abs_high_word(x.y)));
  }
  const int E = block_exponent(hw, ured);
  if (threadIdx.x == 0) we[blockIdx.x] = E;
#pragma unroll
  for (int q = 0; q < 4; q += 2) {
    int q1, q0, p1, p0;
    quantize(a[q], E, q1, q0);
    quantize(a[q + 1], E, p1, p0);
    const int64_t i = e0 / 2 + (q >> 1) * T + threadIdx.x;
    reinterpret_cast<int2*>(w1)[i] = make_int2(q1, p1);
    reinterpret_cast<int2*>(w0)[i] = make_int2(q0, p0);
  }
  nn = block_sum_256(nn, red);
  if (threadIdx.x == 0) part[blockIdx.x] = nn;
}

// (a1 2^29 + a0)(b1 2^29 + b0) added to s[0] 2^58 + s[1] 2^29 + s[2].
__device__ __forceinline__ void fx_add(long long* s, int a1, int a0, int b1, int b0) {
  s[0] += (long long)a1 * b1;
  s[1] += (long long)a1 * b0;
  s[1] += (long long)a0 * b1;
  s[2] += (long long)a0 * b0;
}

// hi 2^64 + lo (signed) times 2^e, rounded to FP64 with integer operations (an
// FP64 conversion by one lane takes the FP64 pipe as long as a full warp's).
// Results below FP64's normal range are zero, those above it infinite.
__device__ __forceinline__ double fx_to_double(long long hi, unsigned long long lo, int e) {
  const bool neg = hi < 0;
  if (neg) {
    lo = ~lo + 1;
    hi = ~hi + (lo == 0 ? 1 : 0);
  }
  if (hi == 0 && lo == 0) return 0.0;
  const int lz = hi ? __clzll(hi) : 64 + __clzll((long long)lo);
  unsigned long long top;  // the 64 leading bits
  if (lz >= 64) top = lo << (lz - 64);
  else top = lz ? ((unsigned long long)hi << lz) | (lo >> (64 - lz)) : (unsigned long long)hi;
  const int be = 127 - lz + e + 1023;
  if (be <= 0) return 0.0;
  if (be >= 2047) return __longlong_as_double(0x7FF0000000000000LL | (neg ? 1LL << 63 : 0));
  const unsigned long long m = (top >> 11) + ((top >> 10) & 1);  // in [2^52, 2^53]
  const unsigned long long bits = ((unsigned long long)be << 52) + (m - (1ULL << 52));
  return __longlong_as_double((long long)(bits | (neg ? 1ULL << 63 : 0)));
}

// A 128-bit sum: three 64-bit sums hold 32 products (fx_add), longer ones are folded into it.
struct Acc128 {
  unsigned long long lo;
  long long hi;
  __device__ __forceinline__ void add(unsigned long long l, long long h) {
    lo += l;
    hi += h + (lo < l ? 1 : 0);
  }
  // + (s[0] 2^58 + s[1] 2^29 + s[2]) / 2^shift, rounded down
  __device__ __forceinline__ void fold(const long long* s, int shift = 0) {
    const __int128 t = (((__int128)s[0] << 58) + ((__int128)s[1] << 29) + s[2]) >> shift;
    add((unsigned long long)t, (long long)(t >> 64));
  }
  // the sum over the warp, as FP64 times 2^e
  __device__ __forceinline__ double warp_sum(int e) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      add(__shfl_xor_sync(0xffffffffu, lo, o), __shfl_xor_sync(0xffffffffu, hi, o));
    return fx_to_double(hi, lo, e);
  }
};

// The 128-bit sum over the warp as FP64 times 2^e.
__device__ __forceinline__ double fx_warp_sum(const long long* s, int e) {
  Acc128 a{0, 0};
  a.fold(s);
  return a.warp_sum(e);
}

// Full pass, dots: h2[k] = conj(V_k) w' for k in [0, nk) from the planes. A block
// takes one tile and DOT_GROUP vectors, one per warp at a time, DOT_LOADS 16-byte
// loads of each plane in flight per lane. Blocks of one tile are adjacent, so that
// the tiles read last still have their Q1 planes in L2 when k_update_q starts with
// them. The last block of a group sums its vectors' tile partials (part[k][tile]).
// LOCAL (256-entry tiles): the block forms its tile of w' and the planes of it
// itself, one entry per thread, and the tile's first block writes the |w'|^2
// partial; else the tile's planes come from k_local (L1 after the first warp).
// Two vectors per warp (w read once for both) measured slower: 157 us
// (80 registers, 37 % of the warps).
// 647,079 rows, 100 vectors: 95 us (5.5 TB/s) at two loads of each plane and five
// blocks per SM; one load and eight blocks 96, four loads and four blocks 114.
constexpr int DOT_GROUP = 8;
constexpr int DOT_LOADS = 2;
constexpr int DOT_MINB = 5;

// What the tile of w' is made from (LOCAL) or where k_local left it.
struct WTile {
  const double* vj;
  const double* w;
  const double2* apart;  // partials of h_j
  int na;
  const int* w1;
  const int* w0;
  int* we;               // [ntile] exponents of w' (LOCAL writes them)
  double* npart;         // [ntile] partials of |w'|^2 (LOCAL writes them)
};

template <int TILE, bool LOCAL>
__global__ void __launch_bounds__(256, DOT_MINB)
    k_dots_q(const int* Q1, const int* Q0, const int* E, int64_t ld, int ntile, int64_t n, int nk, int ngroups,
             WTile W, double* part, Scal S, int j) {
  pdl_begin();
  static_assert(!LOCAL || TILE == 256, "one entry per thread");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int tile = (int)(blockIdx.x / (unsigned)ngroups), g = (int)(blockIdx.x % (unsigned)ngroups);
  const int ka = g * DOT_GROUP, kb = min(nk, ka + DOT_GROUP);
  const int64_t e0 = (int64_t)tile * TILE;
  constexpr int U = TILE / 128 < DOT_LOADS ? TILE / 128 : DOT_LOADS;
  const int k = ka + wid;
  const int stop = S.flags[0];
  const int4* a1 = reinterpret_cast<const int4*>(W.w1 + e0) + lane;
  const int4* a0 = reinterpret_cast<const int4*>(W.w0 + e0) + lane;
  const int64_t row = k < kb ? k : ka;  // a warp without a vector reads the group's first
  const int4* v1 = reinterpret_cast<const int4*>(Q1 + row * ld + e0) + lane;
  const int4* v0 = reinterpret_cast<const int4*>(Q0 + row * ld + e0) + lane;
  int ex = E[row * ntile + tile] - 112;
  int4 x1[U], x0[U];
#pragma unroll
  for (int u = 0; u < U; u++) {
    x1[u] = __ldcg(v1 + 32 * u);
    x0[u] = __ldcs(v0 + 32 * u);
  }
  __shared__ __align__(16) int sw[2][LOCAL ? TILE : 4];
  if (LOCAL) {
    __shared__ double red[8];
    __shared__ unsigned ured[8];
    __shared__ double2 s_h;
    const int64_t i = e0 + threadIdx.x;
    double x = 0.0, u = 0.0, y = 0.0, v = 0.0;  // this double and the other part of its entry
    if (i < n) {
      x = W.w[i];
      u = W.vj[i];
      y = W.w[i ^ 1];
      v = W.vj[i ^ 1];
    }
    if (stop) return;
    if (wid == 0) {
      const double2 t = sum_partials(W.apart, W.na);
      if (lane == 0) {
        s_h = t;
        if (blockIdx.x == 0) S.alpha[j] = t.x;
      }
    }
    __syncthreads();
    const double2 h = s_h;
    const bool im = threadIdx.x & 1;
    const double2 t = three_term(im ? make_double2(y, x) : make_double2(x, y),
                                 im ? make_double2(v, u) : make_double2(u, v), h);
    x = im ? t.y : t.x;
    const int ew = block_exponent(abs_high_word(x), ured);
    ex += ew;
    int q1, q0;
    quantize(x, ew, q1, q0);
    sw[0][threadIdx.x] = q1;
    sw[1][threadIdx.x] = q0;
    if (g == 0) {
      const double nn = block_sum_256(x * x, red);  // the whole block
      if (threadIdx.x == 0) {
        W.npart[tile] = nn;
        W.we[tile] = ew;
      }
    }
    __syncthreads();
    a1 = reinterpret_cast<const int4*>(sw[0]) + lane;
    a0 = reinterpret_cast<const int4*>(sw[1]) + lane;
  } else {
    ex += W.we[tile];
    if (stop) return;
  }
  if (k < kb) {
    long long s[2][3];  // (re, im)
#pragma unroll
    for (int c = 0; c < 2; c++) s[c][0] = s[c][1] = s[c][2] = 0;
#pragma unroll 1
    for (int t = 0; t < TILE / 4; t += 32 * U) {
      if (t) {
#pragma unroll
        for (int u = 0; u < U; u++) {
          x1[u] = __ldcg(v1 + t + 32 * u);
          x0[u] = __ldcs(v0 + t + 32 * u);
        }
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int4 b1 = a1[t + 32 * u], b0 = a0[t + 32 * u];
        fx_add(s[0], x1[u].x, x0[u].x, b1.x, b0.x);
        fx_add(s[0], x1[u].y, x0[u].y, b1.y, b0.y);
        fx_add(s[0], x1[u].z, x0[u].z, b1.z, b0.z);
        fx_add(s[0], x1[u].w, x0[u].w, b1.w, b0.w);
        // Im conj(v) w = vr wi - vi wr
        fx_add(s[1], x1[u].x, x0[u].x, b1.y, b0.y);
        fx_add(s[1], -x1[u].y, -x0[u].y, b1.x, b0.x);
        fx_add(s[1], x1[u].z, x0[u].z, b1.w, b0.w);
        fx_add(s[1], -x1[u].w, -x0[u].w, b1.z, b0.z);
      }
    }
#pragma unroll
    for (int c = 0; c < 2; c++) {
      const double d = fx_warp_sum(s[c], ex);
      if (lane == 0) part[((int64_t)k * ntile + tile) * 2 + c] = d;
    }
  }
  if (!last_block(S.cnt + CNT_DOTS + g, ntile)) return;
  if (k < kb) {
    double a = 0, b = 0;
    const double* p = part + (int64_t)k * ntile * 2;
    for (int t = lane; t < ntile; t += 32) {
      a += __ldcg(p + (int64_t)t * 2);
      b += __ldcg(p + (int64_t)t * 2 + 1);
    }
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      S.h2[2 * k] = a;
      S.h2[2 * k + 1] = b;
    }
  }
}

// A tile's values v (thread t holds entries t, t + NT, ...) into row k of the
// planes: exponent, then the fixed-point parts, zeros past the vector's end.
template <int TILE, int NT, int NE>
__device__ __forceinline__ void store_planes(const double (&v)[NE], unsigned hw, int64_t tile, int* q1, int* q0, int* E,
                                             unsigned* ured) {
  const int ex = block_exponent(hw, ured);
  if (threadIdx.x == 0) E[tile] = ex;
#pragma unroll
  for (int q = 0; q < NE; q++) {
    const int i = q * NT + threadIdx.x;
    if (TILE % NT == 0 || i < TILE) {
      int p1, p0;
      quantize(v[q], ex, p1, p0);
      q1[tile * TILE + i] = p1;
      q0[tile * TILE + i] = p0;
    }
  }
}

// (hi, lo) FP32 pair of x, hi = x rounded to nearest even, lo = the rest rounded,
// hi + lo = x to 2^-48, from the bit pattern (the FP64 pipe's conversions would
// cost as much as the rest of k_update_q's epilogue). |x| < 2^-74 gives zeros
// (below 2^-74 of a normalized vector).
__device__ __forceinline__ float2 split_f64(double x) {
  const long long b = __double_as_longlong(x);
  const int ex = (int)((b >> 52) & 0x7FF) - 1023;
  const long long m = (b & 0xFFFFFFFFFFFFFLL) | 0x10000000000000LL;  // 53 bits
  const int hi = (int)((m + (1LL << 28) - 1 + ((m >> 29) & 1)) >> 29);  // 24 bits, ties to even
  const int lo = (int)(m - ((long long)hi << 29));
  if (ex < -74) return make_float2(0.f, 0.f);
  const unsigned sg = (unsigned)(b >> 32) & 0x80000000u;
  const float sh = __uint_as_float(sg | (unsigned)(ex - 23 + 127) << 23);
  const float sl = __uint_as_float(sg | (unsigned)(ex - 52 + 127) << 23);
  return make_float2((float)hi * sh, (float)lo * sl);
}

// One vector entry: V_{j+1} and its split for the next SpMV (double-float xs, or fixed
// point xq below 2^xe).
__device__ __forceinline__ void store_entry(double v, int64_t i, double* vout, float2* xs, int2* xq, int xe) {
  vout[i] = v;
  if (xs) xs[i] = split_f64(v);
  if (xq) xq[i] = fix_scaled(v, xe);
}

// Where v_{j+1} goes: its row of V, of the planes, and the SpMV's split input.
struct NextVec {
  double* v;
  float2* xs;
  int2* xq;
  int* xe;  // the exponent xq is below
  int* q1;
  int* q0;
  int* E;
};

// Full pass, correction, and the next vector: v_{j+1} = (w' - sum_k h2[k] V_k) /
// beta_{j+1} with its planes. One block per tile; KS slices of the vectors share
// it, each thread four entries: KS = 1 (256 threads, 4 KB runs per vector) where
// the tiles alone give every SM two blocks (gs_step_q), else 1024 threads (KS = 4, or 16
// on 256-entry tiles). Tiles are taken in descending order (see k_dots_q).
// LOCAL: w' = w - h_j v_j is formed here (see k_dots_q), else k_local left it in w.
// A pass with a coefficient not below 2^-30 |w'| (near an invariant subspace)
// subtracts in FP64 and takes the norm of the result; its last block then scales
// the whole vector.
template <int TILE, int KS, bool LOCAL>
__global__ void __launch_bounds__(KS * TILE / 4) k_update_q(const double* V, const int* Q1, const int* E, int64_t ld,
                                                            int ntile, int64_t n, int nk, WTile W, double* w,
                                                            double* part, Scal S, int j, double breakdown_tol,
                                                            NextVec nx) {
  pdl_begin();
  constexpr int NT = KS * TILE / 4, TP = TILE / 4;
  constexpr int NE = (TILE + NT - 1) / NT;  // entries per thread after the sum over slices
  extern __shared__ float hf[];  // [2 nk] coefficients times the tile's scale
  __shared__ double red1[NT / 32];
  __shared__ unsigned ured[NT / 32];
  __shared__ __align__(16) float sred[KS * TILE];
  __shared__ double s_inv, s_hh, s_nn;
  __shared__ double2 s_h;
  __shared__ int s_hexp;  // exponent of the largest coefficient
  __shared__ int s_wexp, s_xe;  // of the largest |w'|; of the next SpMV's input
  const int tile = (int)(gridDim.x - 1 - blockIdx.x);
  const int64_t r0 = (int64_t)tile * TILE;
  const int stop = S.flags[0];
  double a[NE];
  double wo[NE], vo[NE], vp[NE];  // LOCAL: the entry's other part, v_j's two parts
#pragma unroll
  for (int q = 0; q < NE; q++) {
    const int i = q * NT + threadIdx.x;
    const bool in = i < TILE && r0 + i < n;
    a[q] = in ? w[r0 + i] : 0.0;
    if (LOCAL) {
      vo[q] = in ? W.vj[r0 + i] : 0.0;
      wo[q] = in ? w[(r0 + i) ^ 1] : 0.0;
      vp[q] = in ? W.vj[(r0 + i) ^ 1] : 0.0;
    }
  }
  for (int t = threadIdx.x; t < 2 * nk; t += NT) {
    const int e = E[(int64_t)(t >> 1) * ntile + tile] - 27;  // value = q1 2^(E - 56 + 29)
    const double h = S.h2[t];
    // |h| 2^e below FP32's range is below 2^-100 of the tile's entries: zero
    hf[t] = e < -126 ? 0.0f : f64_lead_f32(h) * __uint_as_float((unsigned)(e + 127) << 23);
  }
  if (stop) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (wid == 0) {
    double hh = 0;
    unsigned hw = 0;
    for (int t = lane; t < 2 * nk; t += 32) {
      const double h = S.h2[t];
      hh += h * h;
      hw = max(hw, abs_high_word(h));
    }
    hh = warp_sum(hh);
    hw = __reduce_max_sync(0xffffffffu, hw);
    if (lane == 0) {
      s_hh = hh;
      s_hexp = (int)(hw >> 20) - 1023;
    }
  } else if (wid == 1) {
    const double nn = sum_partials(W.npart, ntile);
    if (lane == 0) s_nn = nn;
  } else if (wid == 3) {
    int e = -1023;
    for (int t = lane; t < ntile && nx.xq; t += 32) e = max(e, __ldcg(W.we + t));
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) s_wexp = e;
  } else if (LOCAL && wid == 2) {
    const double2 h = sum_partials(W.apart, W.na);
    if (lane == 0) s_h = h;
  }
  __syncthreads();  // hf too
  // the correction is summed in FP32 only while every coefficient is below 2^-30 |w'|
  // (by exponents: (2^(e+1))^2 <= 2^(E-60), 2^E <= |w'|^2)
  const bool small = 2 * (s_hexp + 2) <= (int)(abs_high_word(s_nn) >> 20) - 1023 - 60;
  if (LOCAL) {
    const double2 h = s_h;
#pragma unroll
    for (int q = 0; q < NE; q++) {
      const bool im = threadIdx.x & 1;  // NT is even: every entry of this thread is the same part
      const double2 t = three_term(im ? make_double2(wo[q], a[q]) : make_double2(a[q], wo[q]),
                                   im ? make_double2(vp[q], vo[q]) : make_double2(vo[q], vp[q]), h);
      a[q] = im ? t.y : t.x;
    }
  }
  if (tile == 0 && threadIdx.x == 0) S.alpha[j] += S.h2[2 * j];
  if (small) {
    if (threadIdx.x == 0) {
      const double b2 = s_nn - s_hh;
      s_inv = rsqrt(b2);
      if (nx.xq) {
        s_xe = scaled_exponent(s_wexp, s_hh, s_inv);
        if (tile == 0) *nx.xe = s_xe;
      }
      if (tile == 0) beta_from(S, j, b2, breakdown_tol);
    }
    const int sl = (int)threadIdx.x / TP, pos = (int)threadIdx.x % TP;
    const int4* p = reinterpret_cast<const int4*>(Q1 + r0) + pos;
    const int64_t ld4 = ld / 4;
    float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int k = sl; k < nk; k += KS) {
      const int4 v = __ldcg(p + k * ld4);
      const float v0 = (float)v.x, v1 = (float)v.y, v2 = (float)v.z, v3 = (float)v.w;
      const float hr = hf[2 * k], hi = hf[2 * k + 1];
      d[0] = fmaf(hr, v0, fmaf(-hi, v1, d[0]));
      d[1] = fmaf(hr, v1, fmaf(hi, v0, d[1]));
      d[2] = fmaf(hr, v2, fmaf(-hi, v3, d[2]));
      d[3] = fmaf(hr, v3, fmaf(hi, v2, d[3]));
    }
    *reinterpret_cast<float4*>(sred + sl * TILE + pos * 4) = make_float4(d[0], d[1], d[2], d[3]);
    __syncthreads();
    const double inv = s_inv;
    const int xe = s_xe;
    unsigned hw = 0;
#pragma unroll
    for (int q = 0; q < NE; q++) {
      const int i = q * NT + threadIdx.x;
      if (i < TILE && r0 + i < n) {
        float c = 0.f;
#pragma unroll
        for (int z = 0; z < KS; z++) c += sred[z * TILE + i];
        a[q] = (a[q] - (double)c) * inv;
        store_entry(a[q], r0 + i, nx.v, nx.xs, nx.xq, xe);
        hw = max(hw, abs_high_word(a[q]));
      }
    }
    store_planes<TILE, NT>(a, hw, tile, nx.q1, nx.q0, nx.E, ured);
    return;
  }
  double nn = 0;
  unsigned hw = 0;
#pragma unroll
  for (int q = 0; q < NE; q++) {
    const int64_t r = r0 + q * NT + threadIdx.x;
    if (q * NT + (int)threadIdx.x >= TILE || r >= n) continue;
    for (int k = 0; k < nk; k++) {
      const double v = V[k * n + r], u = V[k * n + (r ^ 1)], hr = S.h2[2 * k], hi = S.h2[2 * k + 1];
      a[q] -= (r & 1) ? hr * v + hi * u : hr * v - hi * u;
    }
    nx.v[r] = a[q];  // not yet scaled (w is still read by other blocks' three-term step)
    nn += a[q] * a[q];
    hw = max(hw, abs_high_word(a[q]));
  }
  nn = block_sum_256(nn, red1);
  hw = block_max(hw, ured);
  if (threadIdx.x == 0) {
    part[tile] = nn;
    nx.E[tile] = (int)hw;  // the tile's exponent goes here at the end
  }
  if (!last_block(S.cnt + CNT_UPDATE, gridDim.x)) return;
  double s = 0;
  hw = 0;
  for (int t = threadIdx.x; t < (int)gridDim.x; t += NT) {
    s += __ldcg(part + t);
    hw = max(hw, (unsigned)__ldcg(nx.E + t));
  }
  s = block_sum_256(s, red1);
  hw = block_max(hw, ured);
  if (threadIdx.x == 0) {
    s_inv = rsqrt(s);
    s_xe = scaled_exponent(word_exponent(hw), 0.0, s_inv);
    if (nx.xq) *nx.xe = s_xe;
    beta_from(S, j, s, breakdown_tol);
  }
  __syncthreads();
  const double inv = s_inv;
  const int xe = s_xe;
  for (int t = 0; t < ntile; t++) {
    hw = 0;
#pragma unroll
    for (int q = 0; q < NE; q++) {
      const int64_t i = (int64_t)t * TILE + q * NT + threadIdx.x;
      a[q] = 0.0;
      if (q * NT + (int)threadIdx.x < TILE && i < n) {
        a[q] = __ldcg(nx.v + i) * inv;
        store_entry(a[q], i, nx.v, nx.xs, nx.xq, xe);
        hw = max(hw, abs_high_word(a[q]));
      }
    }
    store_planes<TILE, NT>(a, hw, t, nx.q1, nx.q0, nx.E, ured);
    __syncthreads();  // ured is written again
  }
}

// The planes of the start vector. One block of TILE / 4 threads per tile.
template <int TILE>
__global__ void __launch_bounds__(TILE / 4) k_planes_q(const double* src, int64_t n, NextVec nx) {
  pdl_begin();
  constexpr int NT = TILE / 4;
  __shared__ unsigned ured[NT / 32];
  double a[4];
  unsigned hw = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int64_t i = (int64_t)blockIdx.x * TILE + q * NT + threadIdx.x;
    a[q] = i < n ? src[i] : 0.0;
    hw = max(hw, abs_high_word(a[q]));
  }
  store_planes<TILE, NT>(a, hw, blockIdx.x, nx.q1, nx.q0, nx.E, ured);
}
