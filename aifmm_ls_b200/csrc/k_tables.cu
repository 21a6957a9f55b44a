// k_tables.cu -- leaf-level interaction tables by adaptive Gauss-Legendre
// quadrature on the GPU (one CTA per Hankel or Bessel factor, explicit depth-first stack).
//
// Replaces the reference's precomputation, which is what getMatrixEntry reads
// for a uniform tree (only the leaf level's tables are ever used):
//  * far field: C(n, l) = r^2 int_{[-1,1]^2} J_n(kappa r |P|) e^{-in theta_P} T_a(x) T_b(y) dP
//    (LS/FarFieldInteraction.hpp:62-74, 115-135), M = C Q^+ (:152-160)
//  * near field, 9 colleague directions: V(i, l) = int H0(kappa r |X_i - P|) T_a T_b dP
//    (LS/NearFieldInteraction1.hpp:98-128), table = (i r^2/4) V Q^+ (LS/LS_Assembly.hpp:1290-1317)
//  * quadrature: LS/domain2D.hpp:46-138 -- a panel is split in four; the parent is
//    accepted when |I_parent - sum I_child| < 1e-7, otherwise every child is refined;
//    the result is the sum of accepted panels' own estimates in depth-first order.
#include "kernels.h"
#include "smem_limit.h"

namespace {

struct QuadParams {
  int n_cheb, rank, nb;       // nb = degree (degree + 1) / 2
  double kappa, r;            // wavenumber, leaf half width
  const double* gl_x;         // 10 Gauss-Legendre nodes (reference order)
  const double* gl_w;
  const int2* basis;          // (a, b) per basis function
  const double* cheb;         // n_cheb 1-D Chebyshev nodes
  double2* C;                 // 121 x nb (column-major)
  double2* V;                 // 9 * rank x nb  (row = dir * rank + i)
  int* status;                // nonzero on stack overflow / panel budget exhausted
};

__device__ double cheb_T(double x, int n) { return cos(n * acos(x)); }

// J_n(x) for a single order n >= 0 (x >= 0)
__device__ double jn_single(int n, double x) {
  if (x == 0.0) return n == 0 ? 1.0 : 0.0;
  if (x <= 8.0) {
    // power series: sum_k (-1)^k (x/2)^{2k+n} / (k! (n+k)!)
    double lead = 1.0, h = 0.5 * x;
    for (int k = 1; k <= n; ++k) lead *= h / k;
    double t = lead, s = lead, q = -h * h;
    for (int k = 1; k < 200; ++k) {
      t *= q / ((double)k * (double)(n + k));
      s += t;
      if (fabs(t) < 1e-18 * fabs(s)) break;
    }
    return s;
  }
  if (n < x) {
    double a = j0(x), b = j1(x);
    if (n == 0) return a;
    for (int k = 1; k < n; ++k) { double c = (2.0 * k / x) * b - a; a = b; b = c; }
    return b;
  }
  int N = (int)(fmax((double)n, x) + 24.0 + 10.0 * cbrt(fmax((double)n, x)));
  N += (N & 1);
  double jp1 = 0.0, jc = 1e-250, norm = 2.0 * jc, want = 0.0;
  for (int k = N; k >= 1; --k) {
    double jm = ((2.0 * k) / x) * jc - jp1;
    jp1 = jc; jc = jm;
    if (((k - 1) & 1) == 0) norm += (k - 1 == 0 ? 1.0 : 2.0) * jm;
    if (k - 1 == n) want = jm;
    if (fabs(jc) > 1e200) { jc *= 1e-200; jp1 *= 1e-200; norm *= 1e-200; want *= 1e-200; }
  }
  return want / norm;
}

// The factor of an integrand that does not depend on the basis function: task = order
// + 60 (FAR), or direction * rank + node.
template <bool FAR>
__device__ double2 base_value(const QuadParams& P, int task, double x, double y) {
  if (FAR) {
    const int nn = task - 60;
    // these sums of squares keep one rounding each: the 6-digit noise of zeros shows it
    const double R2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));
    const double normX = sqrt(R2);
    const double argJ = P.kappa * P.r * normX;
    const double th = atan2(y, x);
    const int m = nn < 0 ? -nn : nn;
    double jv = jn_single(m, argJ);
    if (nn < 0 && (m & 1)) jv = -jv;
    double s, c;
    sincos((double)m * th, &s, &c);
    // exp(-I n theta) = (cos(n theta), -sin(n theta))
    double2 e = make_double2(c, nn >= 0 ? -s : s);
    return make_double2(jv * e.x, jv * e.y);
  } else {
    const int rank = P.rank, n = P.n_cheb;
    const int dir = task / rank, i = task % rank;
    const double Nc[9][2] = {{-2, -2}, {0, -2}, {2, -2}, {2, 0}, {2, 2}, {0, 2}, {-2, 2}, {-2, 0}, {0, 0}};
    const double cbx = Nc[dir][0] * P.r, cby = Nc[dir][1] * P.r;
    const double ax = P.r * P.cheb[i % n] + 0.0, ay = P.r * P.cheb[i / n] + 0.0;
    const double Xx = (ax - cbx) / P.r, Xy = (ay - cby) / P.r;
    const double dx = Xx - x, dy = Xy - y;
    const double R2 = __fma_rn(dx, dx, __dmul_rn(dy, dy));
    const double R = sqrt(R2);
    const double arg = P.kappa * P.r * R;
    return make_double2(j0(arg), y0(arg));
  }
}

constexpr int kStack = 160;
constexpr int kWarps = 4;

// Shared memory of quad_kernel: the stack's integrals (kStack x nb), the four children's
// integrals, their 100 base values and Chebyshev values, then the panels.
__host__ __device__ inline size_t quad_smem_bytes(int nb, int degree) {
  return sizeof(double2) * ((size_t)kStack * nb + 4 * (size_t)nb + 4 * 100) + sizeof(double) * (4 * 2 * 10 * (size_t)degree) +
         sizeof(double4) * kStack + sizeof(unsigned long long) * kStack;
}

// All basis functions of one base factor in one CTA.  The integrals of the basis
// functions refine different panels of the same dyadic tree: a panel is visited for
// those (mask) whose parent panel was refused, in the depth-first order of each, and
// its base values -- Bessel functions, what an evaluation costs -- serve all of them.
// Warp c evaluates child c of the panel on top: the lanes share its 100 points, then
// lane l sums basis function l over the points in the reference's (m, n) order.
// What bounds it: the longest depth-first chain (the panels around a node).  6 x 6
// nodes, 21 basis functions: near 0.36 ms (one warp per integral: 1.84 ms), far 0.055
// (0.17) ms.
template <bool FAR>
__global__ void __launch_bounds__(32 * kWarps) quad_kernel(QuadParams P, int degree, double eps) {
  extern __shared__ double2 qsm[];
  const int nb = P.nb, task = blockIdx.x;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double2* sI = qsm;                       // kStack x nb
  double2* child = sI + (size_t)kStack * nb;  // 4 x nb
  double2* buf = child + 4 * nb + 100 * w; // this warp's base values
  double* cheb0 = reinterpret_cast<double*>(child + 4 * nb + 400);
  double* Tx = cheb0 + w * 20 * degree;    // T_a at the 10 abscissae
  double* Ty = Tx + 10 * degree;
  double4* pan = reinterpret_cast<double4*>(cheb0 + 80 * degree);  // (xc, yc, xr, yr)
  unsigned long long* mask = reinterpret_cast<unsigned long long*>(pan + kStack);
  __shared__ int s_top, s_fail;
  __shared__ unsigned long long s_refine;
  // the panel's integrals of the basis functions in `todo` into out[l]; one warp
  auto panel = [&](double xc, double yc, double xr, double yr, unsigned long long todo, double2* out) {
    for (int p = lane; p < 100; p += 32) {
      const int m = p / 10, n = p % 10;
      buf[p] = base_value<FAR>(P, task, xc + xr * P.gl_x[m], yc + yr * P.gl_x[n]);
    }
    for (int e = lane; e < 10 * degree; e += 32) {
      const int a = e / 10, m = e % 10;
      Tx[e] = cheb_T(xc + xr * P.gl_x[m], a);
      Ty[e] = cheb_T(yc + yr * P.gl_x[m], a);
    }
    __syncwarp();
    for (int l = lane; l < nb; l += 32) {
      if (!((todo >> l) & 1)) continue;
      const int2 ab = P.basis[l];
      double2 s = make_double2(0.0, 0.0);
      for (int m = 0; m < 10; ++m) {
        const double ta = Tx[ab.x * 10 + m], wm = P.gl_w[m];
#pragma unroll
        for (int n = 0; n < 10; ++n) {
          const double tb = Ty[ab.y * 10 + n], wt = wm * P.gl_w[n];
          const double2 h = buf[m * 10 + n];
          // each product and sum rounded by itself, as when the values pass through memory
          s.x = __dadd_rn(s.x, __dmul_rn(wt, __dmul_rn(__dmul_rn(h.x, ta), tb)));
          s.y = __dadd_rn(s.y, __dmul_rn(wt, __dmul_rn(__dmul_rn(h.y, ta), tb)));
        }
      }
      const double a = xr * yr;
      out[l] = make_double2(s.x * a, s.y * a);
    }
  };
  const unsigned long long all = nb == 64 ? ~0ull : (1ull << nb) - 1;
  if (w == 0) {
    panel(0.0, 0.0, 1.0, 1.0, all, sI);
    if (lane == 0) {
      pan[0] = make_double4(0.0, 0.0, 1.0, 1.0);
      mask[0] = all;
      s_top = 1;
      s_fail = 0;
    }
  }
  // lane l of warp 0 keeps the accepted sum of basis functions l and l + 32
  double2 acc[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
  long budget[2] = {400000, 400000};
  __syncthreads();
  for (;;) {
    const int top = s_top - 1;
    if (top < 0 || s_fail) break;
    const double4 pa = pan[top];
    const unsigned long long mk = mask[top];
    const double hx = 0.5 * pa.z, hy = 0.5 * pa.w;
    // children in the order (-,-), (+,-), (+,+), (-,+)
    const double cx = pa.x + (w == 1 || w == 2 ? hx : -hx), cy = pa.y + (w >= 2 ? hy : -hy);
    panel(cx, cy, hx, hy, mk, child + w * nb);
    __syncthreads();
    if (w == 0) {
      unsigned long long refine = 0;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int l = lane + 32 * u;
        bool r = false;
        if (l < nb && ((mk >> l) & 1)) {
          const double2 I = sI[(size_t)top * nb + l];
          double2 err = I;
          for (int c = 0; c < 4; ++c) err = csub(err, child[c * nb + l]);
          if (--budget[u] <= 0 || top + 4 > kStack) s_fail = 1;
          if (hypot(err.x, err.y) < eps) acc[u] = cadd(acc[u], I);
          else r = true;
        }
        refine |= (unsigned long long)__ballot_sync(0xffffffffu, r) << (32 * u);
      }
      if (lane == 0) {
        s_refine = refine;
        s_top = refine && top + 4 <= kStack ? top + 4 : top;
      }
    }
    __syncthreads();
    const unsigned long long refine = s_refine;
    if (refine && top + 4 <= kStack) {  // child c goes to top + 3 - c: child 0 is next
      const int at = top + 3 - w;
      for (int l = lane; l < nb; l += 32) sI[(size_t)at * nb + l] = child[w * nb + l];
      if (lane == 0) {
        pan[at] = make_double4(cx, cy, hx, hy);
        mask[at] = refine;
      }
    }
    __syncthreads();
  }
  if (w == 0) {
    if (lane == 0 && s_fail) atomicExch(P.status, 1);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int l = lane + 32 * u;
      if (l >= nb) continue;
      if (FAR) {
        const double rr = P.r * P.r;
        P.C[task + (size_t)l * 121] = make_double2(rr * acc[u].x, rr * acc[u].y);
      } else {
        P.V[(size_t)task * nb + l] = acc[u];  // row-major V[dir*rank + i][l]
      }
    }
  }
}

// Q (rank x nb) Chebyshev Vandermonde at the leaf nodes, Q^+ = (Q^T Q)^{-1} Q^T by
// Cholesky (Q has orthogonal columns on tensor Chebyshev nodes, so this is benign).
// One CTA.
__global__ void tables_finish_kernel(QuadParams P, double* qpinv_out) {
  extern __shared__ double sm[];
  const int rank = P.rank, nb = P.nb, n = P.n_cheb;
  double* Q = sm;                    // rank x nb
  double* G = Q + rank * nb;         // nb x nb
  double* Qp = G + nb * nb;          // nb x rank
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int t = tid; t < rank * nb; t += nt) {
    int i = t % rank, l = t / rank;
    int2 ab = P.basis[l];
    Q[i + l * rank] = cheb_T(P.cheb[i % n], ab.x) * cheb_T(P.cheb[i / n], ab.y);
  }
  __syncthreads();
  for (int t = tid; t < nb * nb; t += nt) {
    int a = t % nb, b = t / nb;
    double s = 0.0;
    for (int i = 0; i < rank; ++i) s += Q[i + a * rank] * Q[i + b * rank];
    G[a + b * nb] = s;
  }
  __syncthreads();
  if (tid == 0) {  // Cholesky G = L L^T in place (lower)
    for (int k = 0; k < nb; ++k) {
      double d = G[k + k * nb];
      for (int p = 0; p < k; ++p) d -= G[k + p * nb] * G[k + p * nb];
      d = sqrt(d);
      G[k + k * nb] = d;
      for (int i = k + 1; i < nb; ++i) {
        double s = G[i + k * nb];
        for (int p = 0; p < k; ++p) s -= G[i + p * nb] * G[k + p * nb];
        G[i + k * nb] = s / d;
      }
    }
  }
  __syncthreads();
  for (int col = tid; col < rank; col += nt) {  // solve G x = Q^T e_col
    double x[64];
    for (int a = 0; a < nb; ++a) x[a] = Q[col + a * rank];
    for (int a = 0; a < nb; ++a) {
      double s = x[a];
      for (int p = 0; p < a; ++p) s -= G[a + p * nb] * x[p];
      x[a] = s / G[a + a * nb];
    }
    for (int a = nb - 1; a >= 0; --a) {
      double s = x[a];
      for (int p = a + 1; p < nb; ++p) s -= G[p + a * nb] * x[p];
      x[a] = s / G[a + a * nb];
    }
    for (int a = 0; a < nb; ++a) Qp[a + col * nb] = x[a];
  }
  __syncthreads();
  for (int t = tid; t < nb * rank; t += nt) qpinv_out[t] = Qp[t];
}

// M = C Q^+ and near = (V * i r^2 / 4) Q^+, one thread per entry: 9 us at 6 x 6 nodes,
// where the one CTA that also inverts took 0.17 ms for both (the inverse takes 0.07)
__global__ void tables_product_kernel(QuadParams P, const double* __restrict__ Qp, double2* M, double2* nearT) {
  const int rank = P.rank, nb = P.nb;
  const int nM = 121 * rank, t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nM) {
    const int r = t % 121, j = t / 121;
    double2 s = make_double2(0.0, 0.0);
    for (int l = 0; l < nb; ++l) {
      double2 c = P.C[r + (size_t)l * 121];
      double qv = Qp[l + j * nb];
      s.x += c.x * qv; s.y += c.y * qv;
    }
    M[r + (size_t)j * 121] = s;
    return;
  }
  const int u = t - nM;
  if (u >= 9 * rank * rank) return;
  const double rB = P.r;
  const int dir = u / (rank * rank), rem = u % (rank * rank);
  const int i = rem % rank, j = rem / rank;
  double2 s = make_double2(0.0, 0.0);
  for (int l = 0; l < nb; ++l) {
    double2 v = P.V[((size_t)dir * rank + i) * nb + l];
    // ((V * I) * r) * r / 4  (LS_Assembly.hpp:1313)
    double2 vt = make_double2(-v.y, v.x);
    vt.x = vt.x * rB; vt.y = vt.y * rB;
    vt.x = vt.x * rB; vt.y = vt.y * rB;
    vt.x = vt.x / 4.0; vt.y = vt.y / 4.0;
    double qv = Qp[l + j * nb];
    s.x += vt.x * qv; s.y += vt.y * qv;
  }
  nearT[(size_t)dir * rank * rank + i + (size_t)j * rank] = s;
}

// ---- the 6-digit text round trip (printf "%.6g", strtod) in exact integer arithmetic
//
// |v| = m 2^q, and D = |v| 10^p rounded half to even is the six-digit decimal, p such
// that 10^5 <= |v| 10^p < 10^6.  The value read back is D / 10^p rounded to nearest: one
// IEEE division for p <= 22 (both are exact doubles), else a long division by 5^p to the
// result's bits, a guard and a sticky bit.  Up to p = 54, m 5^p fits 192 bits; the tiny
// rows of M (J_60 of a small argument) take p up to 328 and words in local memory.
// 32,040 values: 62 us, against 8.7 ms of snprintf and strtod on the host.
// Magnitudes from 9e5 up, which no table holds, are left to the host (return false).
typedef unsigned long long u64;
typedef unsigned __int128 u128;
struct Fives {
  u128 v[55];
  double ten[23];
  constexpr Fives() : v(), ten() {
    v[0] = 1;
    for (int i = 1; i < 55; ++i) v[i] = v[i - 1] * 5;
    ten[0] = 1.0;
    for (int i = 1; i < 23; ++i) ten[i] = ten[i - 1] * 10.0;
  }
};
__constant__ Fives c_five = Fives();

constexpr int kWords = 28;  // 32-bit words: 2^53 5^330 and 2^(1 + log2 5^330) fit

// m 5^p as words, low first; returns how many are in use
__device__ __noinline__ int five_words(u64 m, int p, unsigned* N) {
  int n = 0;
  for (; m; m >>= 32) N[n++] = (unsigned)m;
  for (; p > 0; p -= 13) {
    const unsigned f = (unsigned)c_five.v[p < 13 ? p : 13];
    u64 carry = 0;
    for (int i = 0; i < n; ++i) {
      carry += (u64)N[i] * f;
      N[i] = (unsigned)carry;
      carry >>= 32;
    }
    if (carry) N[n++] = (unsigned)carry;
  }
  return n;
}

// m 5^p 2^-sh: the whole part, its next bit and whether anything is set below that
__device__ u64 scaled_wide(u64 m, int p, int sh, bool* half, bool* below) {
  unsigned N[kWords];
  const int n = five_words(m, p, N);
  auto word = [&](int i) { return i < n ? (u64)N[i] : 0ull; };
  const int w = sh >> 5, b = sh & 31;  // sh > 0 here
  const u64 D = ((word(w) | word(w + 1) << 32) >> b) | (b ? (word(w + 2) << 32) << (32 - b) : 0ull);
  const int hb = sh - 1;
  *half = (word(hb >> 5) >> (hb & 31)) & 1;
  bool rest = (word(hb >> 5) & ((1u << (hb & 31)) - 1)) != 0;
  for (int i = 0; i < (hb >> 5) && i < n; ++i) rest = rest || N[i];
  *below = rest;
  return D;
}

// D / 10^p to the nearest double (subnormal ones too), D a whole number below 2^20
__device__ double quotient_wide(u64 D, int p) {
  unsigned d[kWords + 1], rem[kWords + 1];
  const int n = five_words(1, p, d) + 1;  // one word of room for the shifts
  d[n - 1] = 0;
  for (int i = 0; i < n; ++i) rem[i] = 0;
  // start with rem = D 2^s as long as 5^p, or one bit less long
  const int dbits = 32 * (n - 1) - __clz(d[n - 2]), Dbits = 64 - __clzll(D);
  int s = dbits - Dbits;
  {
    const int w = s >> 5, b = s & 31;
    const u64 x = D << b;  // below 2^52
    rem[w] = (unsigned)x;
    if (w + 1 < n) rem[w + 1] = (unsigned)(x >> 32);
  }
  auto take = [&]() {  // rem >= d ? subtract it
    for (int i = n - 1; i >= 0; --i) {
      if (rem[i] > d[i]) break;
      if (rem[i] < d[i]) return false;
    }
    long long c = 0;
    for (int i = 0; i < n; ++i) {
      c += (long long)rem[i] - (long long)d[i];
      rem[i] = (unsigned)c;
      c >>= 32;
    }
    return true;
  };
  auto twice = [&]() {
    unsigned c = 0;
    for (int i = 0; i < n; ++i) {
      const unsigned x = rem[i];
      rem[i] = (x << 1) | c;
      c = x >> 31;
    }
  };
  // the leading bit of D / 10^p has the weight 2^lead
  bool bit = take();
  if (!bit) { twice(); ++s; bit = take(); }
  const int lead = -s - p;
  const int nbits = lead >= -1022 ? 53 : lead + 1075;  // of the result
  u64 mant = 0;
  for (int k = 0; k < nbits; ++k) {
    mant = (mant << 1) | (bit ? 1 : 0);
    twice();
    bit = take();
  }
  bool sticky = false;
  for (int i = 0; i < n; ++i) sticky = sticky || rem[i];
  if (bit && (sticky || (mant & 1))) ++mant;
  return ldexp((double)mant, lead - nbits + 1);
}

__device__ bool round6_exact(double v, double* out) {
  *out = v;
  const u64 bits = (u64)__double_as_longlong(v);
  const int be = (int)((bits >> 52) & 0x7ff);
  u64 m = bits & 0xfffffffffffffull;
  if ((bits << 1) == 0 || be == 0x7ff) return true;  // zeros, infinities and NaN stay
  const double av = fabs(v);
  if (!(av < 9e5)) return false;
  if (be) m |= 1ull << 52;
  const int q = (be ? be : 1) - 1075;
  int p = 5 - (int)floor(log10(av));  // off by one at most: corrected by D itself
  u64 D = 0;
  bool up = false, ok = false;
  for (int tries = 0; tries < 3 && !ok; ++tries) {
    if (p < 0 || p > 330) return false;
    const int sh = -(q + p);  // |v| 10^p = m 5^p / 2^sh
    bool half, below;
    if (p > 54) {  // then sh > 32
      D = scaled_wide(m, p, sh, &half, &below);
    } else {
      const u128 lo = (u128)m * (u64)c_five.v[p], mid = (u128)m * (u64)(c_five.v[p] >> 64);
      const u64 n0 = (u64)lo;
      const u128 hi = (lo >> 64) + mid;  // m 5^p = hi 2^64 + n0
      if (sh <= 0) {  // a whole number below 2^20
        D = n0 << -sh;
        half = below = false;
      } else if (sh <= 64) {
        D = sh == 64 ? (u64)hi : (u64)((hi << (64 - sh)) | (n0 >> sh));
        half = (n0 >> (sh - 1)) & 1;
        below = (n0 & ((1ull << (sh - 1)) - 1)) != 0;
      } else if (sh < 192) {
        const int t = sh - 64;  // bits of hi below D
        D = (u64)(hi >> t);
        half = (u64)(hi >> (t - 1)) & 1;
        below = n0 || (hi & (((u128)1 << (t - 1)) - 1)) != 0;
      } else {
        D = 0;
        half = below = false;
      }
    }
    if (D >= 1000000) { --p; continue; }
    if (D < 100000) { ++p; continue; }
    up = half && (below || (D & 1));
    ok = true;
  }
  if (!ok) return false;
  D += up;
  const double r = p <= 22 ? (double)D / c_five.ten[p] : quotient_wide(D, p);
  *out = v < 0.0 ? -r : r;
  return true;
}
__global__ void round6_kernel(double* a, int na, double* b, int nb, int* left) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= na + nb) return;
  double* p = t < na ? a + t : b + (t - na);
  double r;
  if (round6_exact(*p, &r)) *p = r;
  else atomicExch(left, 1);
}

}  // namespace

// Host launcher: all pointers are device pointers.  Returns a CUDA error code.
int aifmm_launch_tables(int n_cheb, int degree, double kappa, double r, const double* gl_x, const double* gl_w,
                        const int2* basis, const double* cheb, double2* Cwork, double2* Vwork, int* status,
                        double* qpinv, double2* M, double2* nearT, cudaStream_t stream) {
  QuadParams P;
  P.n_cheb = n_cheb; P.rank = n_cheb * n_cheb; P.nb = degree * (degree + 1) / 2;
  P.kappa = kappa; P.r = r; P.gl_x = gl_x; P.gl_w = gl_w; P.basis = basis; P.cheb = cheb;
  P.C = Cwork; P.V = Vwork; P.status = status;
  const double eps = 1e-7;  // LS/FarFieldInteraction.hpp:37, LS/NearFieldInteraction1.hpp:112
  const size_t qs = quad_smem_bytes(P.nb, degree);
  if (P.nb > 64 || qs > 220 * 1024) return (int)cudaErrorInvalidValue;
  static SmemLimit attr[3];
  if (const int e = smem_limit(quad_kernel<true>, attr[0])) return e;
  if (const int e = smem_limit(quad_kernel<false>, attr[1])) return e;
  if (const int e = smem_limit(tables_finish_kernel, attr[2])) return e;
  quad_kernel<true><<<121, 32 * kWarps, qs, stream>>>(P, degree, eps);
  quad_kernel<false><<<9 * P.rank, 32 * kWarps, qs, stream>>>(P, degree, eps);
  size_t smem = sizeof(double) * ((size_t)P.rank * P.nb + P.nb * P.nb + P.nb * P.rank);
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  tables_finish_kernel<<<1, 256, smem, stream>>>(P, qpinv);
  const int entries = 121 * P.rank + 9 * P.rank * P.rank;
  tables_product_kernel<<<(entries + 127) / 128, 128, 0, stream>>>(P, qpinv, M, nearT);
  return (int)cudaGetLastError();
}

// The 6-digit text round trip of both tables on the device; *left is set (to be zeroed
// by the caller) if a value is 9e5 or above and keeps its digits.
int aifmm_launch_round6(double2* M, double2* nearT, int rank, int* left, cudaStream_t stream) {
  const int na = 2 * 121 * rank, nb = 2 * 9 * rank * rank;
  round6_kernel<<<(na + nb + 127) / 128, 128, 0, stream>>>(reinterpret_cast<double*>(M), na,
                                                           reinterpret_cast<double*>(nearT), nb, left);
  return (int)cudaGetLastError();
}
