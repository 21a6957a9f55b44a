// entry.cuh -- device evaluation of one Lippmann-Schwinger matrix entry.
//
// Replaces LS2DTree::getMatrixEntry (LS/LS_Assembly.hpp:474-541) reached through
// userkernel::getMatrixEntry (kernel.hpp:130-136):
//   near (leaf j adjacent to leaf i, self included): table(dir)(ii, jj) * kappa^2 q(x_i) (+1 on the diagonal)
//   far: (i/4) kappa^2 q(x_i) sum_{n=-60}^{60} M(n+60, jj) (J_n(R) + i Y_n(R)) e^{i n theta}
//        R = kappa |x_i - c_j|, theta = atan2(x_i - c_j)
//   |entry| < 1e-16 -> 0.
// Bessel functions of integer order replace the reference's per-order Boost
// calls (LS/LS_Assembly.hpp:39-65): J_n by Miller's backward recurrence
// normalised with J_0 + 2 sum J_2k = 1; Y_0, Y_1 from the Neumann series in the
// same J values, then Y_n by forward recurrence.  (CUDA's y0/y1 carry an
// absolute error of ~1e-12 for large arguments, too coarse for 1e-14 entries.)
// The n and -n terms are paired, J_{-n} = (-1)^n J_n, Y_{-n} = (-1)^n Y_n.
#pragma once
#include "common.cuh"
#include "quotient.cuh"

#define AIFMM_SERIES 60

// What bounds an entry: the FP64 pipe, about 4,000 double instructions (busy 52% of the
// time in the ACA, the rest is the latency of the recurrences at 16 warps an SM).
// 592 ACA jobs of 972 x 36 points, ranks 19 to 21: 11.4 ms each way with plain
// divisions and a column of coefficients per lane, 6.2 ms now.  Divisions by R
// and by whole numbers are correctly rounded quotients from a reciprocal
// (quotient.cuh), the counters are doubles (conversions run at a fraction of the FP64 rate),
// and the coefficients are laid out with the sources of a leaf next to each other (Mt:
// the lanes of a warp read neighbouring sources).  Results are those of plain IEEE
// divisions, bit for bit.

// 1 / k
constexpr int kRecips = 1024;
struct RecipTable {
  double r[kRecips];
  constexpr RecipTable() : r() {
    for (int k = 1; k < kRecips; ++k) r[k] = 1.0 / k;
  }
};
static __device__ const RecipTable d_recip = RecipTable();
__device__ __forceinline__ double recip_of(int k) { return k < kRecips ? __ldg(&d_recip.r[k]) : 1.0 / (double)k; }

// Complex products with the fused product of each part named (1: the first, 2: the
// second), as the entry has always been rounded.
template <int X, int Y>
__device__ __forceinline__ double2 cmul_f(double2 a, double2 b) {
  double2 r;
  r.x = X == 1 ? __fma_rn(a.x, b.x, -__dmul_rn(a.y, b.y)) : __fma_rn(-a.y, b.y, __dmul_rn(a.x, b.x));
  r.y = Y == 1 ? __fma_rn(a.x, b.y, __dmul_rn(a.y, b.x)) : __fma_rn(a.y, b.x, __dmul_rn(a.x, b.y));
  return r;
}

// W_n = M_n e^{in theta} + (-1)^n M_{-n} e^{-in theta}   (n >= 1); Mp, Mm: M_n, M_{-n}
template <bool ODD>
__device__ __forceinline__ double2 series_w(const double2* __restrict__ Mp, const double2* __restrict__ Mm, double2 e) {
  const double2 a = cmul_f<1, 1>(__ldg(Mp), e);
  const double2 b = cmul_f<1, 2>(__ldg(Mm), cconj(e));
  return ODD ? csub(a, b) : cadd(a, b);
}

template <bool V>
struct OrderOdd { static constexpr bool value = V; };

// sum_{n=-60}^{60} M_n H_n(R) e^{in th}, M_n = Mc[n ld]
// Pass 1 (downward): Miller's recurrence for J_N..J_0 accumulating sum J_n W_n,
// the normalisation J_0 + 2 sum J_2k and the Neumann sums that give Y_0, Y_1
// (Y_0 = (2/pi)[(ln(R/2)+gamma) J_0 - 2 sum_k (-1)^k J_2k / k],
//  Y_1 = -Y_0' = -(2/(pi R)) J_0 + (2/pi)[(ln(R/2)+gamma) J_1 + sum_k (-1)^k (J_2k-1 - J_2k+1) / k]).
// Orders whose J is below 1e-39 (|J_m(R)| <= (R/2)^m / m!: 5e-40 for order 64 at R = 12,
// 3.5e-40 for order 90 at R = 25) are left out of the three sums: they do not reach the
// last place of one.
// Pass 2 (upward): Y_n by forward recurrence accumulating sum Y_n W_n.
// ENX: the fused product of the real part of pass 1's rotation.
template <int ENX>
__device__ __forceinline__ double2 far_series(double R, double th, const double2* __restrict__ Mc, int ld) {
  constexpr int NS = AIFMM_SERIES;
  double s1, c1;
  sincos(th, &s1, &c1);
  const double2 e1 = make_double2(c1, s1);
  const double2 e1c = cconj(e1);
  // ---- pass 1
  const double big = fmax((double)NS, R);
  int N = (int)(big + 24.0 + 10.0 * cbrt(big));
  N += (N & 1);
  const bool mid = R > kQuotLo && R < kQuotHi;
  const double rR = 1.0 / R;
  const int mfull = !(R > 0.0) ? N : R <= 12.0 ? 64 : R <= 25.0 ? 90 : N;
  double jp1 = 0.0, jcur = 1.0e-250;
  double norm = 2.0 * jcur;                          // N is even
  double S0 = ((N / 2) & 1 ? -jcur : jcur) / (N / 2);  // seed term of sum (-1)^k J_2k / k
  double S1 = 0.0;
  double2 acc = make_double2(0.0, 0.0);
  double k2 = 2.0 * (double)N;  // 2 (m + 1)
  const long long hot = __double_as_longlong(1.0e200);
  auto next = [&]() {  // J_m from J_{m+1}, J_{m+2}
    const double q = mid ? quotient(k2, R, rR) : k2 / R;
    const double jnew = __fma_rn(q, jcur, -jp1);
    jp1 = jcur;
    jcur = jnew;
    k2 -= 2.0;
  };
  auto rescale = [&]() {  // stay in range
    if ((__double_as_longlong(jcur) & 0x7fffffffffffffffLL) > hot) {
      jcur *= 1.0e-200; jp1 *= 1.0e-200; norm *= 1.0e-200;
      acc.x *= 1.0e-200; acc.y *= 1.0e-200; S0 *= 1.0e-200; S1 *= 1.0e-200;
    }
  };
  // the pair of orders m (odd), m - 1: k1 = (m + 1) / 2, k1 - 1 = (m - 1) / 2
  int m = N - 1;
  for (; m > mfull && m > NS + 1; m -= 2) {
    next(); rescale();
    next(); rescale();
  }
  double k1 = 0.5 * (double)(m + 1);
  double y1 = recip_of((m + 1) >> 1);
  double sg = (m & 3) == 3 ? 1.0 : -1.0;  // the sign of (-1)^k1
  auto odd = [&](double y2) {
    const double t = sg * jcur;
    S1 += quotient(t, k1, y1);
    if (m > 1) S1 += quotient(t, k1 - 1.0, y2);
  };
  auto even = [&](double y2) {
    norm += (m == 1 ? 1.0 : 2.0) * jcur;
    if (m > 1) S0 += quotient(-sg * jcur, k1 - 1.0, y2);
  };
  for (; m > NS + 1; m -= 2) {
    const double y2 = recip_of((m - 1) >> 1);
    next(); odd(y2); rescale();
    next(); even(y2); rescale();
    k1 -= 1.0; y1 = y2; sg = -sg;
  }
  double sn, cn;
  sincos((double)NS * th, &sn, &cn);
  double2 en = make_double2(cn, sn);  // e^{i 60 th}
  const double2 *Mp = Mc + (size_t)NS * ld, *Mm = Mc - (size_t)NS * ld;
  {  // m = 61, 60
    const double y2 = recip_of((m - 1) >> 1);
    next(); odd(y2); rescale();
    next(); even(y2);
    const double2 w = series_w<false>(Mp, Mm, en);
    acc.x = fma(jcur, w.x, acc.x); acc.y = fma(jcur, w.y, acc.y);
    rescale();
    k1 -= 1.0; y1 = y2; sg = -sg; m -= 2;
  }
  double2 er[3];  // e^{i 48 th}, e^{i 32 th}, e^{i 16 th}
#pragma unroll
  for (int blk = 0; blk < 4; ++blk) {
    // orders 59 .. 48, 47 .. 32, 31 .. 16, 15 .. 0
    if (blk > 0) {
      sincos((double)(m + 1) * th, &sn, &cn);
      en = er[blk - 1] = make_double2(cn, sn);
    }
    for (int stop = 48 - 16 * blk; m > stop; m -= 2) {
      const double y2 = recip_of((m - 1) >> 1);
      next(); odd(y2);
      en = cmul_f<ENX, 2>(en, e1c);  // e^{i m th}
      Mp -= ld; Mm += ld;
      double2 w = series_w<true>(Mp, Mm, en);
      acc.x = fma(jcur, w.x, acc.x); acc.y = fma(jcur, w.y, acc.y);
      rescale();
      next(); even(y2);
      en = cmul_f<ENX, 2>(en, e1c);
      Mp -= ld; Mm += ld;
      w = m == 1 ? __ldg(Mp) : series_w<false>(Mp, Mm, en);
      acc.x = fma(jcur, w.x, acc.x); acc.y = fma(jcur, w.y, acc.y);
      rescale();
      k1 -= 1.0; y1 = y2; sg = -sg;
    }
  }
  const double inorm = 1.0 / norm;
  const double2 SJ = make_double2(acc.x * inorm, acc.y * inorm);
  const double J0 = jcur * inorm, J1 = jp1 * inorm;
  S0 *= inorm; S1 *= inorm;
  const double kTwoOverPi = 0.63661977236758134307553505349;
  const double kEuler = 0.57721566490153286060651209008;
  const double lg = log(0.5 * R) + kEuler;
  double ym = kTwoOverPi * __fma_rn(lg, J0, -2.0 * S0);
  double yc = __fma_rn(kTwoOverPi, __fma_rn(lg, J1, S1), __dmul_rn(__ddiv_rn(-kTwoOverPi, R), J0));
  // ---- pass 2
  const double2 w0 = __ldg(Mc);
  double2 SY = make_double2(ym * w0.x, ym * w0.y);
  double2 e = e1;
  const double inv = 2.0 / R;
  Mp = Mm = Mc;
  double nd = 1.0;
  auto up = [&](auto is_odd) {
    Mp += ld; Mm -= ld;
    const double2 w = series_w<decltype(is_odd)::value>(Mp, Mm, e);
    SY.x = fma(yc, w.x, SY.x); SY.y = fma(yc, w.y, SY.y);
    const double yn = __fma_rn(nd * inv, yc, -ym);
    ym = yc; yc = yn;
    e = cmul_f<1, 1>(e, e1);
    nd += 1.0;
  };
#pragma unroll
  for (int blk = 0; blk < 4; ++blk) {
    // orders 1 .. 15, 16 .. 31, 32 .. 47, 48 .. 60
    if (blk > 0) {
      e = er[3 - blk];
      up(OrderOdd<false>());
    }
    for (int n = 16 * blk + 1; n < (blk == 3 ? 60 : 16 * blk + 15); n += 2) {
      up(OrderOdd<true>());
      up(OrderOdd<false>());
    }
    if (blk < 3) up(OrderOdd<true>());
  }
  // sum (J_n + i Y_n) W_n = SJ + i SY
  return make_double2(SJ.x - SY.y, SJ.y + SY.x);
}

__device__ __forceinline__ int near_dir(int dx, int dy) {
  // neighbour numbering of FMM2DTree (0=(-1,-1) 1=(0,-1) 2=(1,-1) 3=(1,0) 4=(1,1)
  // 5=(0,1) 6=(-1,1) 7=(-1,0)) and 8 = self, the index of LS_Assembly.hpp's N_centers
  const int tab[9] = {0, 1, 2, 7, 8, 3, 6, 5, 4};
  return tab[(dy + 1) * 3 + (dx + 1)];
}

// Entries below it are zero (LS_Assembly.hpp:536-538).
constexpr double kEntryFloor = 1e-16;
// Whether every far entry of a row with the contrast qi is below half of `floor`
__device__ __forceinline__ bool far_is_zero(double qi, const EntryCtx& c, double floor) {
  return c.kappa * c.kappa * fabs(qi) * __ldg(c.far_bound) < 0.5 * floor;
}

// PHI = true: the system matrix A (findPhi, LS_Assembly.hpp:506-511, 528-533);
// PHI = false: the bare integral operator G of the same entry (no kappa^2 q(x_i)
// factor, no identity), the operator the reference applies to the solution to
// get the scattered field (hybrid.cpp:263-281).
// ENX: see far_series (the ACA's entries have always fused the other product).
// Entries below kEntryFloor are zero; a far entry whose bound
// kappa^2 |q_i| max_j sum_n |M_nj| |H_n| is below half of `floor` is returned as zero
// without its series.  With the floor of 1e-16 that changes no result: the bound holds
// for every distance (|H_n| decreases), and half leaves room for the rounding of both.
// Rows outside the contrast's support cost one load instead of 61 orders.
template <bool PHI = true, int ENX = 1>
__device__ __forceinline__ double2 lsa_entry(int i, int j, const EntryCtx& c, double floor = kEntryFloor) {
  const int rank = c.rank;
  const int li = i / rank, ii = i - li * rank;
  const int lj = j / rank, jj = j - lj * rank;
  const int2 a = __ldg(&c.leafxy[li]);
  const int2 b = __ldg(&c.leafxy[lj]);
  const int dx = b.x - a.x, dy = b.y - a.y;
  const double qi = __ldg(&c.q[i]);
  if (dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1) {
    const int dir = near_dir(dx, dy);
    double2 e = __ldg(&c.nearT[(size_t)dir * rank * rank + ii + (size_t)jj * rank]);
    if (PHI) {
      // entry*kappa*kappa*q evaluated left to right (LS_Assembly.hpp:508)
      e.x = e.x * c.kappa; e.y = e.y * c.kappa;
      e.x = e.x * c.kappa; e.y = e.y * c.kappa;
      e.x = e.x * qi; e.y = e.y * qi;
      if (i == j) e.x = 1.0 + e.x;
    }
    if (hypot(e.x, e.y) < kEntryFloor) e = make_double2(0.0, 0.0);
    return e;
  }
  if (PHI && far_is_zero(qi, c, floor)) return make_double2(0.0, 0.0);
  const double2 ri = __ldg(&c.pts[i]);
  const double2 cj = __ldg(&c.leafc[lj]);
  const double ddy = ri.y - cj.y, ddx = ri.x - cj.x;
  const double th = atan2(ddy, ddx);
  const double R = c.kappa * sqrt(__fma_rn(ddy, ddy, __dmul_rn(ddx, ddx)));
  double2 s = far_series<ENX>(R, th, c.Mt + (size_t)AIFMM_SERIES * rank + jj, rank);
  // *= I/4 (exact), then *= kappa*kappa*q (LS_Assembly.hpp:529-531)
  s = make_double2(-0.25 * s.y, 0.25 * s.x);
  if (PHI) {
    const double kq = c.kappa * c.kappa * qi;
    s.x *= kq; s.y *= kq;
    if (i == j) s.x += 1.0;
  }
  if (hypot(s.x, s.y) < kEntryFloor) s = make_double2(0.0, 0.0);
  return s;
}
