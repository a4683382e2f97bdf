// Eigenpairs of the Lanczos tridiagonal T (diagonal a, off-diagonal b[1..m-1]).
//
// Every step of a Sturm count and of a triangular solve waits for the one before it,
// and an FP64 instruction of one warp takes ~64 clocks whether one lane or 32 need it:
// the time is the number of dependent FP64 instructions. So: counts with b^2 squared
// once and comparisons on integers; counting rounds replaced by FP32 pairs where the
// outcome can be checked in one FP64 round; all that is no recurrence spread over the
// warp. The values are those of the plain recurrences (krylov.cuh), bit for bit: in
// sectors with a degenerate ground state the vector depends on the last bit of these.
#pragma once
#include <cfloat>
#include "krylov.cuh"

// Dynamic shared memory: [a | b^2 | FP32 pairs of a | of b^2] with level 4, the first
// two with level 2; level 0 reads global memory.
struct Tri {
  const double* a;
  const double* b2;  // null at level 0
  const double* b;   // global memory
  const float2* fa;  // null below level 4
  const float2* fb;
  int m;
  double glo, ghi, pm, sc;  // Gershgorin interval, smallest pivot, 2^k with the interval * 2^k inside (-1, 1)
};

__device__ __forceinline__ double tri_pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// Stages T (all threads of the block); gersh of krylov.cuh, its maxima over the lanes.
__device__ __forceinline__ Tri tri_stage(const double* a, const double* b, int m, int level) {
  extern __shared__ double tri_sm[];
  Tri T{};
  T.a = a;
  T.b = b;
  T.m = m;
  const int lane = threadIdx.x & 31;
  double l = a[0], h = a[0], bm = 0;
  for (int i = lane; i < m; i += 32) {
    const double v = a[i], bi = i > 0 ? b[i] : 0;
    const double r = (i > 0 ? fabs(bi) : 0) + (i + 1 < m ? fabs(b[i + 1]) : 0);
    l = fmin(l, v - r);
    h = fmax(h, v + r);
    if (i > 0) bm = fmax(bm, bi * bi);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    l = fmin(l, __shfl_xor_sync(0xffffffffu, l, o));
    h = fmax(h, __shfl_xor_sync(0xffffffffu, h, o));
    bm = fmax(bm, __shfl_xor_sync(0xffffffffu, bm, o));
  }
  const double w = fmax(fabs(l), fabs(h));
  T.glo = l - 2 * DBL_EPSILON * w - 1e-300;
  T.ghi = h + 2 * DBL_EPSILON * w + 1e-300;
  T.pm = DBL_MIN * fmax(1.0, bm);
  const int e = ((__double2hiint(w) >> 20) & 0x7ff) - 1022;  // w < 2^e
  if (e > 500 || e < -500) level = level > 2 ? 2 : level;
  T.sc = tri_pow2(level == 4 ? -e - 1 : 0);
  if (level >= 2) {
    double* sa = tri_sm;
    double* sb = tri_sm + m;
    float2* fa = reinterpret_cast<float2*>(tri_sm + 2 * m);
    float2* fb = reinterpret_cast<float2*>(tri_sm + 3 * m);
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
      const double v = a[i], bi = i > 0 ? b[i] : 0;
      sa[i] = v;
      sb[i] = bi * bi;
      if (level == 4) {
        const double vs = v * T.sc, bs = (bi * T.sc) * (bi * T.sc);
        const float vh = (float)vs, bh = (float)bs;
        fa[i] = make_float2(vh, (float)(vs - (double)vh));
        fb[i] = make_float2(bh, (float)(bs - (double)bh));
      }
    }
    __syncthreads();
    T.a = sa;
    T.b2 = sb;
    if (level == 4) {
      T.fa = fa;
      T.fb = fb;
    }
  }
  return T;
}

// sturm_count with b^2 given and its two comparisons on the bits (q is never zero
// when its sign is read).
__device__ __forceinline__ int tri_count(const Tri& T, double x) {
  if (!T.b2) return sturm_count(T.a, T.b, T.m, x, T.pm);
  const long long pmb = __double_as_longlong(T.pm);
  int c = 0;
  double q = T.a[0] - x;
  if ((__double_as_longlong(q) & 0x7fffffffffffffffLL) <= pmb) q = -T.pm;
  c += (unsigned)__double2hiint(q) >> 31;
#pragma unroll 4
  for (int i = 1; i < T.m; i++) {
    q = (T.a[i] - x) - T.b2[i] / q;
    if ((__double_as_longlong(q) & 0x7fffffffffffffffLL) <= pmb) q = -T.pm;
    c += (unsigned)__double2hiint(q) >> 31;
  }
  return c;
}

// Whether an eigenvalue lies below x, in FP32 pairs (~2^-44 of the interval): an
// estimate whose consequences are checked in FP64.
__device__ __forceinline__ bool tri_below_est(const Tri& T, double x) {
  const double xs = x * T.sc;
  const float xh = (float)xs, xl = (float)(xs - (double)xh);
  bool neg = false;
  float qh = 0.f, ql = 0.f;
#pragma unroll 4
  for (int i = 0; i < T.m; i++) {
    const float2 A = T.fa[i], B = T.fb[i];
    float t = 0.f, t2 = 0.f;
    if (i > 0) {
      const float r = __fdividef(1.f, qh);
      t = B.x * r;
      t2 = fmaf(-t, ql, fmaf(-t, qh, B.x) + B.y) * r;
    }
    float d, de, q, qe;
    two_sum(A.x, -xh, d, de);
    two_sum(d, -t, q, qe);
    qe += (de + (A.y - xl)) - t2;
    qh = q + qe;
    ql = qe - (qh - q);
    if (fabsf(qh) < 1e-30f) {
      qh = -1e-30f;
      ql = 0.f;
    }
    neg |= qh < 0.f;
  }
  return neg;
}

constexpr int TRI_THREADS = 128;

// 32-point multisection of [lo, hi] for the lowest eigenvalue to 2 ulp, at most maxit
// rounds (call by the whole block; the result is warp 0's). A round is one FP64 count:
// 11 from the Gershgorin interval. With FP32 pairs at hand the block first narrows an
// estimate to 2^-42 of the interval (128 points a round, a seventh of an FP64 round's
// time), plays the rounds that it decides and checks all of their outcomes in one FP64
// count (the count is monotone in x, so the points next to the crossing decide a round);
// what is wrong or too close to call is left to plain rounds.
__device__ __forceinline__ void tri_multisect(const Tri& T, double& lo, double& hi, int maxit) {
  const int lane = threadIdx.x & 31;
  const double scale = fmax(fabs(T.glo), fabs(T.ghi)), del = scale * 0x1p-42;
  int it = 0;
  if (T.fa && hi - lo > 64 * del) {  // uniform over the block
    double el = lo, eh = hi;
    for (int k = 0; k < 8 && eh - el > del; k++) {
      const double step = (eh - el) * (1.0 / (TRI_THREADS + 1));
      const int n = __syncthreads_count(tri_below_est(T, el + step * (threadIdx.x + 1)));
      const int f = TRI_THREADS - n;  // the first point with an eigenvalue below it
      const double nl = f > 0 ? el + step * f : el;
      if (f < TRI_THREADS) eh = el + step * (f + 1);
      el = nl;
    }
    if (threadIdx.x >= 32) return;
    const double est = 0.5 * (el + eh);
    double pl = lo, ph = hi, keep_lo = 0, keep_hi = 0, y = lo;
    int n = 0, want = -1;
    for (; n < 16 && n < maxit; n++) {
      if (ph - pl <= 2 * DBL_EPSILON * fmax(fabs(pl), fabs(ph))) break;
      const double x = pl + (ph - pl) * (lane + 1) / 33.0;
      if (__any_sync(0xffffffffu, fabs(x - est) <= 2 * del)) break;
      const unsigned hit = __ballot_sync(0xffffffffu, x > est);
      const int f = hit ? __ffs(hit) - 1 : 32;
      const double xf = __shfl_sync(0xffffffffu, x, f < 32 ? f : 31);
      const double xp = __shfl_sync(0xffffffffu, x, f > 0 ? f - 1 : 0);
      if (f < 32) ph = xf;
      if (f > 0) pl = xp;
      if ((lane >> 1) == n) {
        keep_lo = pl;
        keep_hi = ph;
        if (lane & 1) {
          y = ph;
          want = f < 32 ? 1 : -1;
        } else {
          y = pl;
          want = f > 0 ? 0 : -1;
        }
      }
    }
    const int c = tri_count(T, y);
    const unsigned bad = __ballot_sync(0xffffffffu, want >= 0 && (c >= 1) != (want == 1));
    it = bad ? (__ffs(bad) - 1) >> 1 : n;
    if (it > 0) {
      lo = __shfl_sync(0xffffffffu, keep_lo, 2 * it - 1);
      hi = __shfl_sync(0xffffffffu, keep_hi, 2 * it - 1);
    }
  }
  if (threadIdx.x >= 32) return;
  for (; it < maxit; it++) {
    if (hi - lo <= 2 * DBL_EPSILON * fmax(fabs(lo), fabs(hi))) break;
    const double x = lo + (hi - lo) * (lane + 1) / 33.0;
    const unsigned hit = __ballot_sync(0xffffffffu, tri_count(T, x) >= 1);
    const int f = hit ? __ffs(hit) - 1 : 32;  // first point with an eigenvalue below it
    const double xf = __shfl_sync(0xffffffffu, x, f < 32 ? f : 31);
    const double xp = __shfl_sync(0xffffffffu, x, f > 0 ? f - 1 : 0);
    const double nhi = f < 32 ? xf : hi, nlo = f > 0 ? xp : lo;
    if (nhi == hi && nlo == lo) break;
    hi = nhi;
    lo = nlo;
  }
}

// s / d, correctly rounded, for r the rounded 1 / d (0 when d is outside 2^+-450): one
// correction makes s r a quotient within an ulp, a second one with the exact remainder
// rounds it (P. Markstein, IBM J. Res. Dev. 34, 111 (1990)). Five dependent operations.
__device__ __forceinline__ double tri_div(double s, double d, double r) {
  const unsigned e = (unsigned)(__double2hiint(s) >> 20) & 0x7ffu;
  if (r == 0.0 || e - 573u > 900u) return s / d;
  double q = s * r;
  q = fma(fma(-d, q, s), r, q);
  return fma(fma(-d, q, s), r, q);
}

// tri_inverse_iteration of krylov.cuh by one warp, everything in shared memory (sm: 8 m
// doubles): the recurrences on lane 0 with their values in registers, the rest over the
// lanes. The vector is at sm + 2 m.
__device__ __forceinline__ void tri_inverse_warp(const double* a, const double* b, int m, double lam, double* sm) {
  const int lane = threadIdx.x & 31;
  double *sa = sm, *sb = sm + m, *y = sm + 2 * m, *d = sm + 3 * m, *u1 = sm + 4 * m, *u2 = sm + 5 * m,
         *l = sm + 6 * m;
  int* piv = reinterpret_cast<int*>(sm + 7 * m);
  double anorm = 0;
  for (int i = lane; i < m; i += 32) {
    const double ai = a[i], bi = b[i], bn = i + 1 < m ? b[i + 1] : 0;
    sa[i] = ai;
    sb[i] = bi;
    anorm = fmax(anorm, fabs(ai) + (i ? fabs(bi) : 0) + (i + 1 < m ? fabs(bn) : 0));
    d[i] = ai - lam;
    u1[i] = bn;
    u2[i] = 0;
    y[i] = 1.0 / sqrt((double)m) * (1.0 + 0.01 * (i % 7));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) anorm = fmax(anorm, __shfl_xor_sync(0xffffffffu, anorm, o));
  const double tiny = DBL_EPSILON * fmax(anorm, 1e-300);
  __syncwarp();
  if (lane == 0) {
    double dc = d[0], uc = u1[0];  // row i as it stands
    for (int i = 0; i + 1 < m; i++) {
      const double sub = sb[i + 1], dn = d[i + 1], un = u1[i + 1];
      if (fabs(dc) >= fabs(sub)) {
        const double f = dc != 0 ? sub / dc : 0;
        piv[i] = 0;
        l[i] = f;
        d[i] = dc;
        u1[i] = uc;
        dc = fma(-f, uc, dn);
        uc = un;
      } else {
        const double f = dc / sub;
        piv[i] = 1;
        l[i] = f;
        d[i] = sub;
        u1[i] = dn;
        u2[i] = i + 2 < m ? un : 0;
        dc = fma(-f, dn, uc);
        uc = i + 2 < m ? -f * un : un;
      }
    }
    d[m - 1] = dc;
    u1[m - 1] = uc;
  }
  __syncwarp();
  for (int i = lane; i < m; i += 32) {
    double v = d[i];
    if (fabs(v) < tiny) v = v < 0 ? -tiny : tiny;
    d[i] = v;
    const unsigned e = (unsigned)(__double2hiint(v) >> 20) & 0x7ffu;
    sa[i] = e - 573u > 900u ? 0.0 : 1.0 / v;
  }
  __syncwarp();
  for (int itn = 0; itn < 4; itn++) {
    double nrm = 0;
    if (lane == 0) {
      double yc = y[0];
      double yn = m > 1 ? y[1] : 0;
      for (int i = 0; i + 1 < m; i++) {
        const double f = l[i], y2 = i + 2 < m ? y[i + 2] : 0;
        if (piv[i]) {
          y[i] = yn;
          yc = fma(-f, yn, yc);
        } else {
          y[i] = yc;
          yc = fma(-f, yc, yn);
        }
        yn = y2;
      }
      double y1 = 0, y2 = 0, s = yc;  // y[i + 1], y[i + 2], the right side of row i
      for (int i = m - 1; i >= 0; i--) {
        const double sn = i > 0 ? y[i - 1] : 0, di = d[i], ri = sa[i], p1 = u1[i], p2 = u2[i];
        if (i + 1 < m) s = fma(-p1, y1, s);
        if (p2 != 0) s = fma(-p2, y2, s);
        const double v = tri_div(s, di, ri);
        y[i] = v;
        y2 = y1;
        y1 = v;
        s = sn;
      }
#pragma unroll 4
      for (int i = 0; i < m; i++) nrm = fma(y[i], y[i], nrm);
    }
    nrm = sqrt(__shfl_sync(0xffffffffu, nrm, 0));
    __syncwarp();
    for (int i = lane; i < m; i += 32) y[i] /= nrm;
    __syncwarp();
  }
  // sign convention: the first component of the largest magnitude positive
  double best = -1;
  int im = m;
  for (int i = lane; i < m; i += 32)
    if (fabs(y[i]) > best) {
      best = fabs(y[i]);
      im = i;
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, im, o);
    if (ob > best || (ob == best && oi < im)) {
      best = ob;
      im = oi;
    }
  }
  if (im < m && y[im] < 0) {
    __syncwarp();
    for (int i = lane; i < m; i += 32) y[i] = -y[i];
  }
  __syncwarp();
}
