// k_dense.cu -- batched small dense complex linear algebra for the bases and the
// hierarchical elimination.
//
//  * Householder QR with column pivoting: the semantics of Eigen's
//    ColPivHouseholderQR as used by FMM2DTree_find_error.hpp (:1535, :1819,
//    :2092, :2477, :2493, :2510): pivot = first remaining column of largest
//    (downdated) norm, LAPACK xGEQP3 norm downdating (LAPACK Working Note 176),
//    reflector G = I - tau v v^H with beta = -sign(Re a_kk) |x|, exactly-nonzero
//    pivot count from the eps-scaled initial column norm, rank() = #|R_ii| >
//    threshold * max|R_ii|, solve() using only the nonzero pivots.
//  * QR solves, explicit Q (householderQ().block(...)).
//  * Partial-pivoting LU solves for the interpolative operators
//    (get_L2P_P2M_box, :1105-1128).
//  * Batched GEMM / GEAM / Frobenius norms.
// One CTA per factorisation; everything else is batched over descriptor lists.
#include <algorithm>
#include <cstring>

#include "dense.cuh"
#include "entry.cuh"

namespace {

template <typename R>
__device__ __forceinline__ R warp_sum(R x) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
template <typename C>
__device__ __forceinline__ C warp_sum2(C x) {
  for (int o = 16; o > 0; o >>= 1) {
    x.x += __shfl_xor_sync(0xffffffffu, x.x, o);
    x.y += __shfl_xor_sync(0xffffffffu, x.y, o);
  }
  return x;
}

template <typename R>
__device__ R block_sum(R x, R* sh) {
  x = warp_sum(x);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0) { R r = 0; for (int w = 0; w < kW; ++w) r += sh[w]; sh[kW] = r; }
  __syncthreads();
  R r = sh[kW];
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------- QR factor
// Blocks that neither the registers nor the shared memory of a CTA hold (qr.cuh): the
// matrix in global memory, one CTA of 32 warps, the norms and the reflector in shared
// memory where they fit.  A pivot step:
//   1. every warp picks the pivot by itself from the norms (no barrier);
//   2. the pivot column changes places, into shared memory too;
//   3. the sum of squares below the diagonal: 256 partial sums, folded in eight groups
//      of 32, then in order; the reflector;
//   4. every warp applies it to two columns at a time;
//   5. the norms are downdated, a thread a column.
// What bounds it: the columns' way from L2 through one SM (a block of 120 x 120 is 230 KB)
// and the chain of a step.  With 8 warps, the norms in global memory, a thread that scans
// them for the pivot and a warp's 32 lanes all downdating one norm: 1.41 ms for 130 x 120
// complex128, 4.74 ms for 200 x 200, 3.68 ms for 200 x 200 complex64; now 0.84, 2.34 and
// 1.55 ms.
constexpr int kQrT = 1024, kQrW = kQrT / 32, kQrSumW = 8;

template <typename C>
__global__ void __launch_bounds__(kQrT) qr_factor_kernel(const QRJob* __restrict__ jobs, int mcap, int ncap) {
  constexpr unsigned full = 0xffffffffu;
  const QRJob J = jobs[blockIdx.x];
  extern __shared__ double2 qr_sm[];
  __shared__ double sh[kQrSumW];
  __shared__ C s_tau;
  __shared__ int s_rank;
  C* const A = static_cast<C*>(J.a);
  const int lda = J.lda;
  C* tau = static_cast<C*>(J.tau);
  int* perm = J.perm;
  const int m = J.m, n = J.n, size = min(m, n);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const bool staged = m <= mcap && n <= ncap;
  C* const sv = reinterpret_cast<C*>(qr_sm);
  double* const nu = staged ? reinterpret_cast<double*>(sv + ((mcap + 1) & ~1)) : J.norms;
  double* const nd = nu + n;
  C* const row = reinterpret_cast<C*>(nu + 2 * ncap);  // row k, for the norms
  for (int j = tid; j < n; j += kQrT) perm[j] = j;
  if (tid == 0) s_rank = 0;
  // initial column norms (one warp per column)
  for (int j = w; j < n; j += kQrW) {
    double s = 0.0;
    for (int i = lane; i < m; i += 32) s += cabs2_p(A[i + (size_t)j * lda]);
    s = warp_sum(s);
    if (lane == 0) { nu[j] = sqrt(s); nd[j] = nu[j]; }
  }
  __syncthreads();
  double maxnorm = 0.0;
  for (int j = lane; j < n; j += 32) maxnorm = fmax(maxnorm, nu[j]);
  for (int o = 16; o > 0; o >>= 1) maxnorm = fmax(maxnorm, __shfl_xor_sync(full, maxnorm, o));
  const double eps = rl<typename cplx<C>::R>::eps;  // the precision of the data
  const double thr_helper = m > 0 ? (maxnorm * eps) * (maxnorm * eps) / m : 0.0;
  const double downdate_thr = sqrt(eps);
  int nzp = size;
  double maxpivot = 0.0;
  for (int k = 0; k < size; ++k) {
    // 1. the largest updated norm among columns k..n-1; norms within kPivotTie of it
    // count as tied: first index wins.  Norms are not negative: their bits order as
    // their values do.
    unsigned hi = 0, lo = 0;
    for (int j = k + lane; j < n; j += 32) {
      const double v = nu[j];
      const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
      if (h > hi || (h == hi && l > lo)) { hi = h; lo = l; }
    }
    const unsigned mh = __reduce_max_sync(full, hi);
    const unsigned ml = __reduce_max_sync(full, hi == mh ? lo : 0u);
    const double cut = __hiloint2double((int)mh, (int)ml) * (1.0 - kPivotTie);
    unsigned first = (unsigned)n;
    for (int j = k + lane; j < n; j += 32)
      if (nu[j] >= cut) { first = (unsigned)j; break; }
    first = __reduce_min_sync(full, first);
    const int big = first < (unsigned)n ? (int)first : k;
    const double nub = nu[big];
    if (nzp == size && nub * nub < thr_helper * (double)(m - k)) nzp = k;
    // 2. columns k and big change places
    C* const ck = A + (size_t)k * lda;
    C* const v = staged ? sv : ck;
    for (int i = tid; i < m; i += kQrT) {
      C* const cb = A + (size_t)big * lda;
      const C y = cb[i];
      if (big != k) { cb[i] = ck[i]; ck[i] = y; }
      if (staged) v[i] = y;
    }
    __syncthreads();
    if (tid == 0 && big != k) {
      double t = nu[k]; nu[k] = nu[big]; nu[big] = t;
      t = nd[k]; nd[k] = nd[big]; nd[big] = t;
      int p = perm[k]; perm[k] = perm[big]; perm[big] = p;
    }
    // 3. reflector for A(k:m, k)
    if (w < kQrSumW) {
      double tail = 0.0;
      for (int i = k + 1 + tid; i < m; i += 32 * kQrSumW) tail += cabs2_p(v[i]);
      tail = warp_sum(tail);
      if (lane == 0) sh[w] = tail;
    }
    const double2 c0 = c2d(v[k]);
    __syncthreads();
    double tail = 0.0;
#pragma unroll
    for (int q = 0; q < kQrSumW; ++q) tail += sh[q];
    double beta;
    if (tail <= DBL_MIN && c0.y * c0.y <= DBL_MIN) {
      beta = c0.x;
      if (tid == 0) s_tau = cplx<C>::mk(0.0, 0.0);
      for (int i = k + 1 + tid; i < m; i += kQrT) {
        ck[i] = cplx<C>::mk(0.0, 0.0);
        if (staged) v[i] = cplx<C>::mk(0.0, 0.0);
      }
    } else {
      beta = sqrt(cabs2_p(c0) + tail);
      if (c0.x >= 0.0) beta = -beta;
      const double2 den = make_double2(c0.x - beta, c0.y);
      if (w == kQrW - 1) {
        const C t = cplx<C>::from(cconj(cdiv(make_double2(beta - c0.x, -c0.y), make_double2(beta, 0.0))));
        if (lane == 0) s_tau = t;
      }
      for (int i = k + 1 + tid; i < m; i += kQrT) {
        const C y = cplx<C>::from(cdiv(c2d(v[i]), den));
        ck[i] = y;
        if (staged) v[i] = y;
      }
    }
    __syncthreads();
    const C t = s_tau;
    if (tid == 0) { ck[k] = cplx<C>::mk(beta, 0.0); tau[k] = t; }
    maxpivot = fmax(maxpivot, fabs(beta));
    // 4. G = I - t v v^H on columns k+1.., then their norms
    for (int j = k + 1 + w; j < n; j += 2 * kQrW) {
      const bool two = j + kQrW < n;
      C* const col[2] = {A + (size_t)j * lda, A + (size_t)(two ? j + kQrW : j) * lda};
      C s[2] = {cplx<C>::mk(0.0, 0.0), cplx<C>::mk(0.0, 0.0)}, wv[2];
      for (int i = k + 1 + lane; i < m; i += 32) {
        const C y = v[i];
        s[0] = cfmac(y, col[0][i], s[0]);
        s[1] = cfmac(y, col[1][i], s[1]);
      }
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          s[q].x += __shfl_xor_sync(full, s[q].x, o);
          s[q].y += __shfl_xor_sync(full, s[q].y, o);
        }
      }
      C rkj[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const C akj = col[q][k];
        wv[q] = cadd(akj, s[q]);
        rkj[q] = csub(akj, cmul_t(t, wv[q]));
      }
      __syncwarp();
      for (int i = k + 1 + lane; i < m; i += 32) {
        const C tv = cmul_t(t, v[i]);
        col[0][i] = csub(col[0][i], cmul_p(tv, wv[0]));
        if (two) col[1][i] = csub(col[1][i], cmul_p(tv, wv[1]));
      }
      if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (q == 1 && !two) break;
          col[q][k] = rkj[q];
          if (staged) row[j + q * kQrW] = rkj[q];
        }
      }
    }
    __syncthreads();
    // 5. LAWN 176 downdate of the norms, a thread a column; -1 marks those to be summed anew
    int again = 0;
    for (int j = k + 1 + tid; j < n; j += kQrT) {
      const double upd = nu[j];
      if (upd != 0.0) {
        const double2 r = c2d(staged ? row[j] : A[k + (size_t)j * lda]);
        double tmp = hypot(r.x, r.y) / upd;
        tmp = (1.0 + tmp) * (1.0 - tmp);
        if (tmp < 0.0) tmp = 0.0;
        const double rr = upd / nd[j];
        const double tmp2 = tmp * rr * rr;
        if (tmp2 <= downdate_thr) {
          nd[j] = -1.0;
          again = 1;
        } else {
          nu[j] = upd * sqrt(tmp);
        }
      }
    }
    if (__syncthreads_or(again)) {
      for (int j = k + 1 + w; j < n; j += kQrW) {
        if (nd[j] >= 0.0) continue;
        double ss = 0.0;
        for (int i = k + 1 + lane; i < m; i += 32) ss += cabs2_p(A[i + (size_t)j * lda]);
        ss = sqrt(warp_sum(ss));
        __syncwarp();
        if (lane == 0) nu[j] = nd[j] = ss;
      }
      __syncthreads();
    }
  }
  const double thr = J.thr > 0.0 ? J.thr : (double)size * eps;
  const double pre = fabs(maxpivot) * thr;
  int rk = 0;
  for (int i = tid; i < nzp; i += kQrT) rk += (cabsd(A[i + (size_t)i * lda]) > pre);
  rk = __reduce_add_sync(full, rk);
  if (lane == 0 && rk) atomicAdd(&s_rank, rk);
  __syncthreads();
  if (tid == 0) {
    J.info[0] = nzp;
    J.info[1] = s_rank;
    if (J.maxpiv) J.maxpiv[0] = maxpivot;
  }
}

// ---------------------------------------------------------------- QR solve
// one warp per right-hand side column, the column in global memory: systems of any size
template <typename C>
__global__ void __launch_bounds__(kT) qr_solve_kernel(const SolveJob* __restrict__ jobs, const int* __restrict__ col_off,
                                                      int njobs, int total_cols) {
  const int gw = blockIdx.x * kW + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (gw >= total_cols) return;
  int lo = 0, hi = njobs - 1;
  while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (col_off[mid] <= gw) lo = mid; else hi = mid - 1; }
  const SolveJob J = jobs[lo];
  const C* Jqr = static_cast<const C*>(J.qr);
  const C* Jtau = static_cast<const C*>(J.tau);
  const C* JB = static_cast<const C*>(J.B);
  const int c = gw - col_off[lo];
  const int m = J.m, n = J.n;
  const int nzp = J.info[0];
  C* x = static_cast<C*>(J.X) + (size_t)c * J.ldx;
  if (nzp == 0) {
    for (int i = lane; i < n; i += 32) x[i] = cplx<C>::mk(0.0, 0.0);
    return;
  }
  C* wv = static_cast<C*>(J.work) + (size_t)c * m;
  for (int i = lane; i < m; i += 32)
    wv[i] = JB ? JB[i + (size_t)c * J.ldb] : cplx<C>::mk(i == c ? 1.0 : 0.0, 0.0);
  __syncwarp();
  // Q^H b with the first nzp reflectors
  for (int k = 0; k < nzp; ++k) {
    const C* v = Jqr + (size_t)k * J.ldq;
    C s = cplx<C>::mk(0.0, 0.0);
    for (int i = k + 1 + lane; i < m; i += 32) s = cfmac(v[i], wv[i], s);
    s = warp_sum2(s);
    const C t = Jtau[k];
    const C w = cadd(wv[k], s);
    __syncwarp();
    for (int i = k + 1 + lane; i < m; i += 32) wv[i] = csub(wv[i], cmul(cmul(t, v[i]), w));
    if (lane == 0) wv[k] = csub(wv[k], cmul(t, w));
    __syncwarp();
  }
  // back substitution with R(0:nzp, 0:nzp), column oriented
  for (int i = nzp - 1; i >= 0; --i) {
    C xi = cplx<C>::from(cdiv(c2d(wv[i]), c2d(Jqr[i + (size_t)i * J.ldq])));
    __syncwarp();
    if (lane == 0) wv[i] = xi;
    for (int l = lane; l < i; l += 32) wv[l] = csub(wv[l], cmul(Jqr[l + (size_t)i * J.ldq], xi));
    __syncwarp();
  }
  for (int i = lane; i < n; i += 32) x[i] = cplx<C>::mk(0.0, 0.0);
  __syncwarp();
  const C alpha = cplx<C>::from(J.alpha);
  for (int i = lane; i < nzp; i += 32) x[J.perm[i]] = cmul(alpha, wv[i]);
}

// The same for up to 32 RPL rows: a column in a warp's registers (row i in lane i mod 32,
// register i / 32), the factor's next column fetched while the one before it is applied.
// Eight columns a CTA read the factor together.
// What bounds it: the chain of a reflector (dot product, its reduction, update) and of a
// row of the back substitution (division, broadcast, update), 0.6 us each.  One column of
// 130 rows, rank 120: 230 us with the column in global memory, 142 us here; 32 columns of
// 200 rows: 498 and 259 us; 300 rows: 878 and 442 us.  Beyond 384 rows (207 registers) the
// kernel above is the faster one.
template <typename C, int RPL>
__global__ void __launch_bounds__(kT) qr_solve_wide_kernel(const SolveJob* __restrict__ jobs,
                                                           const int* __restrict__ col_off, int njobs, int total_cols) {
  constexpr unsigned full = 0xffffffffu;
  const int gw = blockIdx.x * kW + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (gw >= total_cols) return;
  int lo = 0, hi = njobs - 1;
  while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (col_off[mid] <= gw) lo = mid; else hi = mid - 1; }
  const SolveJob J = jobs[lo];
  const C* Jqr = static_cast<const C*>(J.qr);
  const C* Jtau = static_cast<const C*>(J.tau);
  const C* JB = static_cast<const C*>(J.B);
  const int c = gw - col_off[lo];
  const int m = J.m, n = J.n;
  const int nzp = J.info[0];
  C* x = static_cast<C*>(J.X) + (size_t)c * J.ldx;
  if (nzp == 0) {
    for (int i = lane; i < n; i += 32) x[i] = cplx<C>::mk(0.0, 0.0);
    return;
  }
  const C zero = cplx<C>::mk(0.0, 0.0);
  C wv[RPL], nx[RPL];
#pragma unroll
  for (int q = 0; q < RPL; ++q) {
    const int i = lane + 32 * q;
    wv[q] = i >= m ? zero : JB ? JB[i + (size_t)c * J.ldb] : cplx<C>::mk(i == c ? 1.0 : 0.0, 0.0);
  }
  auto fetch = [&](int k) {
    const C* v = Jqr + (size_t)k * J.ldq;
#pragma unroll
    for (int q = 0; q < RPL; ++q) nx[q] = lane + 32 * q < m ? v[lane + 32 * q] : zero;
  };
  auto from_lane = [&](C a, int l) { return C{__shfl_sync(full, a.x, l), __shfl_sync(full, a.y, l)}; };
  // Q^H b with the first nzp reflectors
  fetch(0);
  C tn = Jtau[0];
#pragma unroll
  for (int Q = 0; Q < RPL; ++Q) {
    for (int kk = 0; kk < 32; ++kk) {
      const int k = 32 * Q + kk;
      if (k >= nzp) break;
      C v[RPL];
#pragma unroll
      for (int q = Q; q < RPL; ++q) v[q] = nx[q];
      const C t = tn;
      if (k + 1 < nzp) { fetch(k + 1); tn = Jtau[k + 1]; }
      C s = zero;
#pragma unroll
      for (int q = Q; q < RPL; ++q) {
        const int i = lane + 32 * q;
        if (i > k && i < m) s = cfmac(v[q], wv[q], s);
      }
      s = warp_sum2(s);
      const C w = cadd(from_lane(wv[Q], kk), s);
#pragma unroll
      for (int q = Q; q < RPL; ++q) {
        const int i = lane + 32 * q;
        if (i > k && i < m) wv[q] = csub(wv[q], cmul_p(cmul_t(t, v[q]), w));
      }
      if (lane == kk) wv[Q] = csub(wv[Q], cmul_t(t, w));
    }
  }
  // back substitution with R(0:nzp, 0:nzp), column oriented
  fetch(nzp - 1);
#pragma unroll
  for (int Q = RPL - 1; Q >= 0; --Q) {
    for (int kk = 31; kk >= 0; --kk) {
      const int i = 32 * Q + kk;
      if (i >= nzp) continue;
      C r[RPL];
#pragma unroll
      for (int q = 0; q <= Q; ++q) r[q] = nx[q];
      if (i > 0) fetch(i - 1);
      const C xi = cplx<C>::from(cdiv(c2d(from_lane(wv[Q], kk)), c2d(from_lane(r[Q], kk))));
#pragma unroll
      for (int q = 0; q <= Q; ++q)
        if (lane + 32 * q < i) wv[q] = csub(wv[q], cmul_p(r[q], xi));
      if (lane == kk) wv[Q] = xi;
    }
  }
  for (int i = lane; i < n; i += 32) x[i] = zero;
  __syncwarp();
  const C alpha = cplx<C>::from(J.alpha);
#pragma unroll
  for (int q = 0; q < RPL; ++q)
    if (lane + 32 * q < nzp) x[J.perm[lane + 32 * q]] = cmul_p(alpha, wv[q]);
}

// ---------------------------------------------------------------- form Q
template <typename C>
__global__ void __launch_bounds__(kT) formq_kernel(const FormQJob* __restrict__ jobs, const int* __restrict__ col_off,
                                                   int njobs, int total_cols) {
  const int gw = blockIdx.x * kW + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (gw >= total_cols) return;
  int lo = 0, hi = njobs - 1;
  while (lo < hi) { int mid = (lo + hi + 1) >> 1; if (col_off[mid] <= gw) lo = mid; else hi = mid - 1; }
  const FormQJob J = jobs[lo];
  const C* Jqr = static_cast<const C*>(J.qr);
  const C* Jtau = static_cast<const C*>(J.tau);
  const int c = gw - col_off[lo];
  const int ncols = J.ncols >= 0 ? J.ncols : J.ncols_dev[0];
  if (c >= ncols) return;
  const int m = J.m, size = min(J.m, J.n);
  C* q = static_cast<C*>(J.Q) + (size_t)c * J.ldQ;
  for (int i = lane; i < m; i += 32) q[i] = cplx<C>::mk(i == c ? 1.0 : 0.0, 0.0);
  __syncwarp();
  for (int k = min(size - 1, c); k >= 0; --k) {
    const C* v = Jqr + (size_t)k * J.ldq;
    C s = cplx<C>::mk(0.0, 0.0);
    for (int i = k + 1 + lane; i < m; i += 32) s = cfmac(v[i], q[i], s);
    s = warp_sum2(s);
    const C t = cconj(Jtau[k]);
    const C w = cadd(q[k], s);
    __syncwarp();
    for (int i = k + 1 + lane; i < m; i += 32) q[i] = csub(q[i], cmul(cmul(t, v[i]), w));
    if (lane == 0) q[k] = csub(q[k], cmul(t, w));
    __syncwarp();
  }
}

// ---------------------------------------------------------------- GEMM
// C = alpha sum_t op(A_t) op(B_t) + beta C over a list of products.  A warp owns one
// 8 x 8 sub-tile of C, a CTA WM x WN of them.  The k dimension of all terms is
// walked in chunks of up to tk, which cp.async brings into a ring of NS buffers (tk <=
// 48; NS = 1: products of a single chunk, tk <= 96).  With NS > 1 a second set of as many warps
// fetches, so that its address arithmetic runs beside the products.  Accumulation
// runs over k in increasing order, term after term.
// What bounds it: latency -- the descriptor, the operands' way from L2, the
// instructions that fetch a chunk, and the DMMAs of a sub-tile one after the other
// (four for every 4 of k at 16 cycles each) -- so tiles are small and many: 16 x 16
// for blocks, 32 x 8 for up to 8 right-hand sides; 32 x 32 reads its operands half as
// often, for batches that fill the chip (flush_gemm).
// An operand lies in shared memory as it lies in global memory, contiguous along the
// rows of op = 0's A and op = 1's B, else along k; leading dimensions = 2 (mod 8)
// and = 4 (mod 8) keep the fragment loads free of bank conflicts either way.  Rows and
// columns outside C are not loaded: what they hold reaches only outputs that are not
// written.
constexpr int kGemmTK = 48, kGemmTK1 = 96, kGemmTerms = 64;  // chunk of a ring, of a single buffer
__host__ __device__ constexpr int gemm_ld_row(int t) { return t + 2; }                       // t = 8, 16, 32
__host__ __device__ constexpr int gemm_ld_k(int tk) { return (tk & 7) == 4 ? tk : tk + 4; }  // tk = 0 (mod 4)
__host__ __device__ constexpr int gemm_area(int t, int tk) {
  return tk * gemm_ld_row(t) > t * gemm_ld_k(tk) ? tk * gemm_ld_row(t) : t * gemm_ld_k(tk);
}

__device__ __forceinline__ void cp_async(double2* dst, const double2* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async(float2* dst, const float2* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
// A chunk of one operand, T threads: element (r, k), r < rows (of a tile of TR), k < kc, from
// src[r + k ld] (along_r) or src[k + r ld].
template <typename C, int TR, int T>
__device__ __forceinline__ void gemm_fetch(C* dst, const C* src, int ld, bool along_r, int rows, int kc, int ldk) {
  const int tid = threadIdx.x % T;
  if (along_r) {
    const int r = tid % TR, k0 = tid / TR;
    if (r < rows) {
      const C* s = src + r + (size_t)k0 * ld;
      C* d = dst + k0 * gemm_ld_row(TR) + r;
      const size_t step = (size_t)(T / TR) * ld;
#pragma unroll 3
      for (int k = k0; k < kc; k += T / TR, s += step, d += (T / TR) * gemm_ld_row(TR)) cp_async(d, s);
    }
  } else {
    const int k0 = tid & 15;
    for (int r = tid >> 4; r < rows; r += T / 16) {
      const C* s = src + (size_t)r * ld;
      C* d = dst + r * ldk;
#pragma unroll 3
      for (int k = k0; k < kc; k += 16) cp_async(d + k, s + k);
    }
  }
}
// d += a b for one m8n8k4 FP64 tensor-core product (each lane: one A element,
// one B element, two accumulators)
__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// One 8 x 8 sub-tile of a chunk of kc; element (i, k) of A at i ai + k ak, (k, j) of B
// at k bk + j bj.  complex128: FP64 tensor cores, a complex product as four real
// ones, Cr += Ar Br + (-Ai) Bi and Ci += Ar Bi + Ai Br, k zero-padded to a multiple of
// 4.  Fragments (PTX ISA, mma.m8n8k4 .f64): A row = lane/4, col = lane%4; B row =
// lane%4, col = lane/4; C row = lane/4, cols 2(lane%4) + {0, 1}.
__device__ __forceinline__ void gemm_chunk(const double2* A, const double2* B, int kc, int ai, int ak, int bk, int bj,
                                           int ca, int cb, int lane, double (&cr)[2], double (&ci)[2]) {
  const int kl = lane & 3;
  const double2* a_ = A + (lane >> 2) * ai + kl * ak;
  const double2* b_ = B + kl * bk + (lane >> 2) * bj;
  const double sa = ca ? -1.0 : 1.0, sb = cb ? -1.0 : 1.0;
#pragma unroll 3
  for (int k4 = 0; k4 < kc; k4 += 4, a_ += 4 * ak, b_ += 4 * bk) {
    double2 a = make_double2(0.0, 0.0), b = a;
    if (k4 + kl < kc) { a = *a_; b = *b_; }
    a.y *= sa;
    b.y *= sb;
    dmma884(cr, a.x, b.x);
    dmma884(cr, -a.y, b.y);
    dmma884(ci, a.x, b.y);
    dmma884(ci, a.y, b.x);
  }
}
// The complex64 products of the mixed form: FP32 fused multiply-adds on the CUDA
// cores, the outputs of a lane where the DMMA's accumulators are.
__device__ __forceinline__ void gemm_chunk(const float2* A, const float2* B, int kc, int ai, int ak, int bk, int bj,
                                           int ca, int cb, int lane, float (&cr)[2], float (&ci)[2]) {
  const float2* a_ = A + (lane >> 2) * ai;
  const float2* b_ = B + 2 * (lane & 3) * bj;
#pragma unroll 4
  for (int kk = 0; kk < kc; ++kk) {
    float2 a = a_[kk * ak];
    if (ca) a.y = -a.y;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float2 b = b_[kk * bk + h * bj];
      if (cb) b.y = -b.y;
      const float2 c = cfma(a, b, make_float2(cr[h], ci[h]));
      cr[h] = c.x;
      ci[h] = c.y;
    }
  }
}

// products that travel in the kernel's parameters (kernels.h, GemmOne)
template <int NS>
using GemmInline = Inline<NS == 1 ? kGemmInline * (int)sizeof(GemmOne) : 16>;

template <typename C, int WM, int WN, int NS>
__global__ void __launch_bounds__(32 * WM * WN * (NS == 1 ? 1 : 2)) gemm_kernel(const GemmDesc* __restrict__ ds,
                                                            const GemmTerm* __restrict__ terms,
                                                            const int2* __restrict__ tiles, int tk,
                                                            const __grid_constant__ GemmInline<NS> inl) {
  constexpr int T = 32 * WM * WN, TM = 8 * WM, TN = 8 * WN, LDA = gemm_ld_row(TM), LDB = gemm_ld_row(TN);
  using R = typename cplx<C>::R;
  extern __shared__ double2 gsm_raw[];
  C* ring = reinterpret_cast<C*>(gsm_raw);
  __shared__ GemmTerm st[NS == 1 ? 1 : kGemmTerms];
  pdl_begin();
  int2 tile;
  GemmDesc D;
  GemmTerm one{};
  if (NS == 1 && !ds) {  // products in the parameters: one grid row each
    const GemmOne& P = reinterpret_cast<const GemmOne*>(inl.b)[blockIdx.y];
    if ((int)blockIdx.x >= ((P.m + TM - 1) / TM) * ((P.n + TN - 1) / TN)) return;
    tile = make_int2((int)blockIdx.y, (int)blockIdx.x);
    D.C = P.C; D.ldc = P.ldc; D.m = P.m; D.n = P.n;
    D.alpha = make_double2((double)P.alpha, 0.0);
    D.beta = make_double2((double)P.beta, 0.0);
    D.term0 = 0; D.nterms = P.k > 0 ? 1 : 0;
    one.A = P.A; one.B = P.B; one.lda = P.lda; one.ldb = P.ldb; one.opA = P.op & 1; one.opB = P.op >> 1; one.k = P.k;
  } else {
    tile = __ldg(&tiles[blockIdx.x]);
    D = ds[tile.x];
    if (NS == 1 && D.nterms > 0) one = terms[D.term0];
  }
  const int ldk = gemm_ld_k(tk), offb = gemm_area(TM, tk), stage = offb + gemm_area(TN, tk);
  const int tiles_m = (D.m + TM - 1) / TM;
  const int row0 = (tile.y % tiles_m) * TM, col0 = (tile.y / tiles_m) * TN;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int si = 8 * (warp % WM), sj = 8 * (warp / WM);
  const int rows = min(TM, D.m - row0), cols = min(TN, D.n - col0);
  const bool mine = si < rows && sj < cols;  // else the sub-tile lies outside C
  R cr[2] = {0, 0}, ci[2] = {0, 0};
  auto fetch = [&](const GemmTerm& F, int k0, C* As) {
    const int kc = min(tk, F.k - k0);
    const C* A = static_cast<const C*>(F.A);
    const C* B = static_cast<const C*>(F.B);
    gemm_fetch<C, TM, T>(As, F.opA ? A + k0 + (size_t)row0 * F.lda : A + row0 + (size_t)k0 * F.lda, F.lda, !F.opA, rows,
                         kc, ldk);
    gemm_fetch<C, TN, T>(As + offb, F.opB ? B + col0 + (size_t)k0 * F.ldb : B + k0 + (size_t)col0 * F.ldb, F.ldb,
                         F.opB, cols, kc, ldk);
  };
  auto multiply = [&](const GemmTerm& G, int k0, const C* As) {
    const int ai = G.opA ? ldk : 1, ak = G.opA ? 1 : LDA, bk = G.opB ? LDB : 1, bj = G.opB ? 1 : ldk;
    gemm_chunk(As + si * ai, As + offb + sj * bj, min(tk, G.k - k0), ai, ak, bk, bj, G.opA, G.opB, lane, cr, ci);
  };
  if (NS == 1) {  // at most one term of at most tk
    pdl_wait();
    if (D.nterms > 0) {
      const GemmTerm G = one;
      if (G.k > 0) {
        fetch(G, 0, ring);
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        if (mine) multiply(G, 0, ring);
      }
    }
  } else {
    {
      const int words = min(D.nterms, kGemmTerms) * (int)(sizeof(GemmTerm) / 8);
      const unsigned long long* src = reinterpret_cast<const unsigned long long*>(terms + D.term0);
      for (int e = tid; e < words; e += 2 * T) reinterpret_cast<unsigned long long*>(st)[e] = __ldg(&src[e]);
    }
    __syncthreads();
    pdl_wait();
    auto term = [&](int t) { return t < kGemmTerms ? st[t] : terms[D.term0 + t]; };
    if (tid >= T) {  // the fetching warps: one barrier per chunk, after the chunk has arrived
      int ft = 0, fk = 0, slot = 0, chunks = 0;
      GemmTerm F{};
      if (D.nterms > 0) F = term(0);
      auto next = [&]() {  // one chunk into the next buffer of the ring (none left: an empty group)
        while (ft < D.nterms && fk >= F.k) {
          fk = 0;
          if (++ft < D.nterms) F = term(ft);
        }
        if (ft < D.nterms) {
          fetch(F, fk, ring + slot * stage);
          fk += tk;
          ++chunks;
        }
        if (++slot == NS) slot = 0;
        asm volatile("cp.async.commit_group;\n" ::: "memory");
      };
#pragma unroll
      for (int q = 0; q < NS - 1; ++q) next();
      for (int c = 0; c < chunks; ++c) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(NS >= 2 ? NS - 2 : 0) : "memory");
        __syncthreads();  // chunk c has arrived, and the buffer of chunk c - 1 is free
        next();
      }
      return;
    }
    int slot = 0;
    for (int t = 0; t < D.nterms; ++t) {
      const GemmTerm G = term(t);
      for (int k0 = 0; k0 < G.k; k0 += tk) {
        __syncthreads();
        if (mine) multiply(G, k0, ring + slot * stage);
        if (++slot == NS) slot = 0;
      }
    }
  }
  const bool zero_beta = D.beta.x == 0.0 && D.beta.y == 0.0;
  const C alpha = cplx<C>::from(D.alpha), beta = cplx<C>::from(D.beta);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = si + (lane >> 2), j = sj + 2 * (lane & 3) + h;
    if (i < rows && j < cols) {
      C* c = static_cast<C*>(D.C) + row0 + i + (size_t)(col0 + j) * D.ldc;
      C s;
      s.x = cr[h];
      s.y = ci[h];
      C v = cmul(alpha, s);
      if (!zero_beta) v = cadd(v, cmul(beta, *c));
      *c = v;
    }
  }
}

// ---------------------------------------------------------------- QR solve (registers)
// Eight lanes own one right-hand side: lane q holds rows q, q + 8, ... in registers,
// a CTA of 128 threads takes 16 columns (kSolveCols).  The first nzp columns of the
// factor and tau are staged once per CTA in shared memory; then only shuffles
// synchronise: Q^H b reflector by reflector, column-oriented back substitution with
// R, the column permutation.
// What bounds it: the chain of 2 nzp dependent steps; a reflector's is its dot
// product over eight lanes (three shuffles: the two upper levels of the sum over 32
// rows stay in a lane), tau and the update, about 350 cycles; a scheduler has one warp,
// which issues in 28% of them and waits for a dependent result in most others.  36 x 36, 12 boxes, 8 columns: 15.2 us (a warp per
// column: 20.8 us); 300 boxes: 19 us (36 us).
// Sums run in the order of 32 lanes over the rows (row mod 32), levels 16 to 1.
constexpr int kSolveCols = 16, kSolveT = 8 * kSolveCols;
// rows of a phase (x 8): the rows of earlier phases cost nothing in a forward step
__host__ __device__ constexpr int solve_phase(int rpl) { return (rpl + 5) / 6; }

template <typename C, int RPL, int I0>
__device__ __forceinline__ void solve_forward(const C* F, int ldf, const C* tau, int m, int nzp, int q, C (&b)[RPL]) {
  const unsigned full = 0xffffffffu;  // every lane of a warp runs along
  constexpr int I1 = I0 + solve_phase(RPL) < RPL ? I0 + solve_phase(RPL) : RPL;
  const int kend = min(8 * I1, nzp);
  constexpr bool ahead = RPL <= 12;  // more rows: the registers do not hold two reflectors
  C vn[ahead ? RPL : 1];
  if (ahead) {
#pragma unroll
    for (int t = I0; t < RPL; ++t) vn[t] = 8 * I0 < kend && q + 8 * t < m ? F[(size_t)(8 * I0) * ldf + q + 8 * t] : b[t];
  }
  for (int k = 8 * I0; k < kend; ++k) {
    C v[RPL];
    C s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = cplx<C>::mk(0.0, 0.0);
#pragma unroll
    for (int t = I0; t < RPL; ++t) {
      if (ahead) v[t] = vn[t];
      else if (q + 8 * t < m) v[t] = F[(size_t)k * ldf + q + 8 * t];
      if ((unsigned)(q + 8 * t - k - 1) < (unsigned)(m - k - 1)) s[t & 3] = cfmac(v[t], b[t], s[t & 3]);
    }
    const C tk = tau[k];
    if (ahead && k + 1 < kend) {
#pragma unroll
      for (int t = I0; t < RPL; ++t)
        if (q + 8 * t < m) vn[t] = F[(size_t)(k + 1) * ldf + q + 8 * t];
    }
    C bk = b[I0];
#pragma unroll
    for (int t = I0; t < I1; ++t)
      if (q + 8 * t == k) bk = b[t];
    bk.x = __shfl_sync(full, bk.x, k & 7, 8);
    bk.y = __shfl_sync(full, bk.y, k & 7, 8);
    C z = cadd(cadd(s[0], s[2]), cadd(s[1], s[3]));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      z.x += __shfl_xor_sync(full, z.x, o);
      z.y += __shfl_xor_sync(full, z.y, o);
    }
    // (the complex64 form has always fused the other product here)
    const C tw = sizeof(C) == 16 ? cmul_p(tk, cadd(bk, z)) : cmul_t(tk, cadd(bk, z));
    const C bn = csub(bk, tw);
#pragma unroll
    for (int t = I0; t < RPL; ++t) {
      if ((unsigned)(q + 8 * t - k - 1) < (unsigned)(m - k - 1)) b[t] = csub(b[t], cmul_p(v[t], tw));
      if (t < I1 && q + 8 * t == k) b[t] = bn;
    }
  }
  if constexpr (I1 < RPL) {
    if (nzp > 8 * I1) solve_forward<C, RPL, I1>(F, ldf, tau, m, nzp, q, b);
  }
}
template <typename C, int RPL, int I0>
__device__ __forceinline__ void solve_backward(const C* F, int ldf, const double2* rinv, int nzp, int q, C (&b)[RPL]) {
  const unsigned full = 0xffffffffu;
  constexpr int I1 = I0 + solve_phase(RPL) < RPL ? I0 + solve_phase(RPL) : RPL;
  if constexpr (I1 < RPL) {
    if (nzp > 8 * I1) solve_backward<C, RPL, I1>(F, ldf, rinv, nzp, q, b);
  }
  for (int i = min(nzp, 8 * I1) - 1; i >= 8 * I0; --i) {
    C r[RPL];
#pragma unroll
    for (int t = 0; t < I1; ++t)
      if (q + 8 * t < i) r[t] = F[(size_t)i * ldf + q + 8 * t];
    const double2 ri = rinv[i];
    C bi = b[I0];
#pragma unroll
    for (int t = I0; t < I1; ++t)
      if (q + 8 * t == i) bi = b[t];
    bi.x = __shfl_sync(full, bi.x, i & 7, 8);
    bi.y = __shfl_sync(full, bi.y, i & 7, 8);
    const C xi = cplx<C>::from(cmul_p(c2d(bi), ri));
#pragma unroll
    for (int t = 0; t < I1; ++t) {
      if (q + 8 * t < i) b[t] = csub(b[t], cmul_p(r[t], xi));
      else if (t >= I0 && q + 8 * t == i) b[t] = xi;
    }
  }
}

constexpr int kSolveInline = 30;
using SolveInline = Inline<kSolveInline * sizeof(SolveJob)>;

template <typename C, int RPL>
__global__ void __launch_bounds__(kSolveT) qr_solve_reg_kernel(const SolveJob* __restrict__ jobs,
                                                               const int2* __restrict__ ctas, int early,
                                                               const __grid_constant__ SolveInline inl) {
  extern __shared__ double2 fsm_raw[];
  pdl_begin();
  int2 at;  // job, first column
  SolveJob J;
  if (jobs) {
    at = __ldg(&ctas[blockIdx.x]);
    J = jobs[at.x];
  } else {  // jobs in the parameters: one grid row each
    at = make_int2((int)blockIdx.y, (int)blockIdx.x * kSolveCols);
    J = reinterpret_cast<const SolveJob*>(inl.b)[blockIdx.y];
    if (at.y >= J.nrhs) return;
  }
  // a kept factor (early) is staged while the launch before this one still runs
  if (!early) pdl_wait();
  const C* Jqr = static_cast<const C*>(J.qr);
  const C* Jtau = static_cast<const C*>(J.tau);
  const C* JB = static_cast<const C*>(J.B);
  const int m = J.m, n = J.n, nzp = J.info[0];
  const int tid = threadIdx.x, lane = tid & 31, q = tid & 7, c = at.y + (tid >> 3);
  const int ldf = m | 1;
  // 1 / R_kk in double (a complex64 pivot near 1e-40 has no FP32 reciprocal), so
  // that back substitution only multiplies; then the factor and tau
  double2* rinv = fsm_raw;
  C* F = reinterpret_cast<C*>(rinv + nzp);  // m x nzp, ld = m|1
  C* tau = F + (size_t)ldf * nzp;
  for (int j = tid >> 5; j < nzp; j += kSolveT / 32)
    for (int i = lane; i < m; i += 32) cp_async(&F[i + j * ldf], &Jqr[i + (size_t)j * J.ldq]);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  for (int k = tid; k < nzp; k += kSolveT) {
    tau[k] = Jtau[k];
    rinv[k] = cdiv(make_double2(1.0, 0.0), c2d(Jqr[k + (size_t)k * J.ldq]));
  }
  if (early) pdl_wait();
  C b[RPL];
  const bool mine = c < J.nrhs;
#pragma unroll
  for (int t = 0; t < RPL; ++t) {
    const int i = q + 8 * t;
    b[t] = mine && i < m ? (JB ? JB[i + (size_t)c * J.ldb] : cplx<C>::mk(i == c ? 1.0 : 0.0, 0.0)) : cplx<C>::mk(0.0, 0.0);
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  if (c - (lane >> 3) >= J.nrhs) return;  // the same in a whole warp
  C* x = static_cast<C*>(J.X) + (size_t)c * J.ldx;
  if (nzp > 0) {
    solve_forward<C, RPL, 0>(F, ldf, tau, m, nzp, q, b);
    solve_backward<C, RPL, 0>(F, ldf, rinv, nzp, q, b);
  }
  if (nzp < n) {
    if (mine)
      for (int i = q; i < n; i += 8) x[i] = cplx<C>::mk(0.0, 0.0);
    __syncwarp();
  }
  const C alpha = cplx<C>::from(J.alpha);
#pragma unroll
  for (int t = 0; t < RPL; ++t) {
    const int i = q + 8 * t;
    if (mine && i < nzp) x[J.perm[i]] = cmul(alpha, b[t]);
  }
}

// ---------------------------------------------------------------- GEAM
// Element sizes per descriptor: the arithmetic is complex128, a complex64
// operand is widened on load and a complex64 result rounded on store.
__device__ __forceinline__ double2 ld_any(const void* p, size_t i, int es) {
  return es == 16 ? static_cast<const double2*>(p)[i] : cplx<double2>::from(static_cast<const float2*>(p)[i]);
}
__device__ __forceinline__ void st_any(void* p, size_t i, int es, double2 v) {
  if (es == 16) static_cast<double2*>(p)[i] = v;
  else static_cast<float2*>(p)[i] = cplx<float2>::from(v);
}
constexpr int kGeamInline = 36;
using GeamInline = Inline<kGeamInline * sizeof(GeamDesc)>;
// one grid row per block
__global__ void __launch_bounds__(256) geam_kernel(const GeamDesc* __restrict__ ds, int nd,
                                                   const __grid_constant__ GeamInline inl) {
  pdl_begin();
  bool waited = false;
  for (int b = blockIdx.y; b < nd; b += gridDim.y) {
    const GeamDesc D = ds ? ds[b] : reinterpret_cast<const GeamDesc*>(inl.b)[b];
    if (!waited) {
      pdl_wait();
      waited = true;
    }
    const int tot = D.m * D.n;
    for (int e = blockIdx.x * 256 + threadIdx.x; e < tot; e += gridDim.x * 256) {
      const int j = e / D.m, i = e - j * D.m;
      double2 a = D.opA ? cconj(ld_any(D.A, j + (size_t)i * D.lda, D.esA)) : ld_any(D.A, i + (size_t)j * D.lda, D.esA);
      if (D.rs) a = cscale(a, D.rs[i]);
      if (D.cs) a = cscale(a, D.cs[j]);
      double2 v = cmul(D.alpha, a);
      const size_t ci = i + (size_t)j * D.ldc;
      if (!(D.beta.x == 0.0 && D.beta.y == 0.0)) v = cadd(v, cmul(D.beta, ld_any(D.C, ci, D.esC)));
      st_any(D.C, ci, D.esC, v);
    }
  }
}

// ---------------------------------------------------------------- norms
constexpr int kNormInline = 64;
using NormInline = Inline<kNormInline * sizeof(NormDesc)>;
__global__ void __launch_bounds__(kT) norm_kernel(const NormDesc* __restrict__ ds,
                                                  const __grid_constant__ NormInline inl) {
  pdl_begin();
  const NormDesc D = ds ? ds[blockIdx.x] : reinterpret_cast<const NormDesc*>(inl.b)[blockIdx.x];
  pdl_wait();
  __shared__ double sh[kW + 1];
  double s = 0.0;
  const int tot = D.m * D.n;
  if (D.lda == D.m) {  // contiguous: no division per element
    for (int e = threadIdx.x; e < tot; e += kT) s += cabs2(ld_any(D.A, e, D.es));
  } else {
    for (int e = threadIdx.x; e < tot; e += kT) {
      const int j = e / D.m, i = e - j * D.m;
      s += cabs2(ld_any(D.A, i + (size_t)j * D.lda, D.es));
    }
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) {
    D.out[0] = sqrt(s);  // may be mapped host memory
    __threadfence_system();
  }
}

// ---------------------------------------------------------------- equilibration
// one CTA per block, one thread per column (mode 0) or row (mode 1)
__global__ void __launch_bounds__(kT) equilibrate_kernel(const EquilDesc* __restrict__ ds) {
  const EquilDesc D = ds[blockIdx.x];
  const int cnt = D.mode == 0 ? D.n : D.m, len = D.mode == 0 ? D.m : D.n;
  for (int c = threadIdx.x; c < cnt; c += kT) {
    double q = 0.0;
    for (int e = 0; e < len; ++e) {
      const double2 a = D.mode == 0 ? D.A[e + (size_t)c * D.lda] : D.A[c + (size_t)e * D.lda];
      const double f = D.scale ? D.scale[e] : 1.0;
      q += cabs2(a) * (f * f);
    }
    const double nrm = sqrt(q);
    const bool ok = nrm > 0.0 && nrm < 1e300;
    D.s[c] = ok ? 1.0 / nrm : 1.0;
    D.is[c] = ok ? nrm : 1.0;
  }
}

// ---------------------------------------------------------------- skeleton LU solve
__global__ void __launch_bounds__(kT) skel_lu_kernel(const SkelLUJob* __restrict__ jobs, EntryCtx ctx) {
  const SkelLUJob J = jobs[blockIdx.x];
  const int r = J.r, m = J.m;
  if (r == 0) return;
  double2* D = J.work;             // r x r
  double2* X = J.work + (size_t)r * r;  // r x m
  const int tid = threadIdx.x;
  __shared__ int s_p;
  for (int e = tid; e < r * r; e += kT) {
    int i = e % r, j = e / r;
    // (the two sites have always rounded the entry's rotation differently, see entry.cuh)
    if (J.adjD) D[i + (size_t)j * r] = cconj(lsa_entry<true, 2>(J.rows[j], J.cols[i], ctx));
    else D[i + (size_t)j * r] = lsa_entry<true, 1>(J.rows[i], J.cols[j], ctx);
  }
  for (int e = tid; e < r * m; e += kT) {
    int i = e % r, j = e / r;
    X[i + (size_t)j * r] = J.adjB ? cconj(J.B[j + (size_t)i * J.ldb]) : J.B[i + (size_t)j * J.ldb];
  }
  __syncthreads();
  // LU with partial pivoting (first row of largest modulus), row swaps applied to X
  for (int k = 0; k < r; ++k) {
    if (tid == 0) {
      int p = k; double best = cabsd(D[k + (size_t)k * r]);
      for (int i = k + 1; i < r; ++i) { double v = cabsd(D[i + (size_t)k * r]); if (v > best) { best = v; p = i; } }
      s_p = p;
      J.piv[k] = p;
    }
    __syncthreads();
    const int p = s_p;
    if (p != k) {
      for (int j = tid; j < r; j += kT) { double2 t = D[k + (size_t)j * r]; D[k + (size_t)j * r] = D[p + (size_t)j * r]; D[p + (size_t)j * r] = t; }
      for (int j = tid; j < m; j += kT) { double2 t = X[k + (size_t)j * r]; X[k + (size_t)j * r] = X[p + (size_t)j * r]; X[p + (size_t)j * r] = t; }
    }
    __syncthreads();
    const double2 d = D[k + (size_t)k * r];
    for (int i = k + 1 + tid; i < r; i += kT) {
      if (!(d.x == 0.0 && d.y == 0.0)) D[i + (size_t)k * r] = cdiv(D[i + (size_t)k * r], d);
    }
    __syncthreads();
    for (int e = tid; e < (r - k - 1) * (r - k - 1); e += kT) {
      int i = k + 1 + e % (r - k - 1), j = k + 1 + e / (r - k - 1);
      D[i + (size_t)j * r] = csub(D[i + (size_t)j * r], cmul_f<1, 2>(D[i + (size_t)k * r], D[k + (size_t)j * r]));
    }
    __syncthreads();
  }
  // forward (unit lower) and back substitution, one thread per right-hand side column
  for (int j = tid; j < m; j += kT) {
    double2* x = X + (size_t)j * r;
    for (int i = 0; i < r; ++i) {
      double2 s = x[i];
      for (int l = 0; l < i; ++l) s = csub(s, cmul_f<1, 2>(D[i + (size_t)l * r], x[l]));
      x[i] = s;
    }
    for (int i = r - 1; i >= 0; --i) {
      double2 s = x[i];
      for (int l = i + 1; l < r; ++l) s = csub(s, cmul_f<1, 2>(D[i + (size_t)l * r], x[l]));
      x[i] = cdiv(s, D[i + (size_t)i * r]);
    }
  }
  __syncthreads();
  for (int e = tid; e < r * m; e += kT) {
    int i = e % r, j = e / r;
    if (J.adjX) J.X[j + (size_t)i * J.ldx] = cconj(X[i + (size_t)j * r]);
    else J.X[i + (size_t)j * J.ldx] = X[i + (size_t)j * r];
  }
}

}  // namespace

int aifmm_launch_qr_factor(const QRJob* d_jobs, int njobs, int mmax, int nmax, int es, cudaStream_t s) {
  if (njobs <= 0) return 0;
  if (!valid_es(es)) return (int)cudaErrorInvalidValue;
  // reflector and norms in shared memory; in global memory where a block is too large
  size_t smem = (size_t)es * (((mmax + 1) & ~1) + (size_t)nmax) + 2 * sizeof(double) * (size_t)nmax;
  if (smem > size_t(200) << 10) smem = mmax = nmax = 0;
  static SmemLimit attr[2];
  if (es == 16) {
    if (const int e = smem_limit(qr_factor_kernel<double2>, attr[0])) return e;
    qr_factor_kernel<double2><<<njobs, kQrT, smem, s>>>(d_jobs, mmax, nmax);
  } else {
    if (const int e = smem_limit(qr_factor_kernel<float2>, attr[1])) return e;
    qr_factor_kernel<float2><<<njobs, kQrT, smem, s>>>(d_jobs, mmax, nmax);
  }
  return (int)cudaGetLastError();
}

namespace {
template <typename C>
int launch_solve_reg(const SolveBatch& g, size_t smem, cudaStream_t s) {
  static SmemLimit attr[6];
  SolveInline inl;
  dim3 grid(g.nctas);
  if (!g.d) {
    memcpy(inl.b, g.h, sizeof(SolveJob) * g.njobs);
    grid = dim3(g.nctas, g.njobs);  // nctas: the most CTAs of one job
  }
#define AIFMM_SOLVE_CASE(I, R)                                                                                       \
  if (g.mmax <= 8 * R) {                                                                                             \
    if (const int e = smem_limit(qr_solve_reg_kernel<C, R>, attr[I])) return e;                                      \
    return launch_chain(qr_solve_reg_kernel<C, R>, grid, kSolveT, smem, s, g.d, g.ctas, (int)g.early, inl);          \
  }
  AIFMM_SOLVE_CASE(0, 3) AIFMM_SOLVE_CASE(1, 5) AIFMM_SOLVE_CASE(2, 8) AIFMM_SOLVE_CASE(3, 12)
  AIFMM_SOLVE_CASE(4, 18) AIFMM_SOLVE_CASE(5, 28)
#undef AIFMM_SOLVE_CASE
  return (int)cudaErrorInvalidValue;
}
}  // namespace

int aifmm_solve_cols() { return kSolveCols; }
int aifmm_solve_inline_max() { return kSolveInline; }
int aifmm_launch_qr_solve_reg(const SolveBatch& g, int es, cudaStream_t s) {
  if (g.nctas <= 0) return 0;
  if (!valid_es(es) || (!g.d && g.njobs > kSolveInline)) return (int)cudaErrorInvalidValue;
  const size_t smem = (size_t)es * ((size_t)(g.mmax | 1) * g.nzpmax + (size_t)g.nzpmax) + sizeof(double2) * g.nzpmax + 64;
  return es == 16 ? launch_solve_reg<double2>(g, smem, s) : launch_solve_reg<float2>(g, smem, s);
}

int aifmm_launch_qr_solve(const SolveJob* d_jobs, const int* d_col_off, int njobs, int total_cols, int mmax, int es,
                          cudaStream_t s) {
  if (njobs <= 0 || total_cols <= 0) return 0;
  if (!valid_es(es)) return (int)cudaErrorInvalidValue;
  const int blocks = (total_cols + kW - 1) / kW;
  // up to kSolveWideMax rows the column stays in registers (the jobs' `work` may be nullptr)
#define AIFMM_SOLVE_WIDE(R)                                                                                     \
  if (mmax <= 32 * R) {                                                                                         \
    if (es == 16) qr_solve_wide_kernel<double2, R><<<blocks, kT, 0, s>>>(d_jobs, d_col_off, njobs, total_cols); \
    else qr_solve_wide_kernel<float2, R><<<blocks, kT, 0, s>>>(d_jobs, d_col_off, njobs, total_cols);           \
    return (int)cudaGetLastError();                                                                             \
  }
  AIFMM_SOLVE_WIDE(4) AIFMM_SOLVE_WIDE(8) AIFMM_SOLVE_WIDE(12)
#undef AIFMM_SOLVE_WIDE
  static_assert(kSolveWideMax == 32 * 12, "the largest case above");
  if (es == 16) qr_solve_kernel<double2><<<blocks, kT, 0, s>>>(d_jobs, d_col_off, njobs, total_cols);
  else qr_solve_kernel<float2><<<blocks, kT, 0, s>>>(d_jobs, d_col_off, njobs, total_cols);
  return (int)cudaGetLastError();
}

int aifmm_launch_formq(const FormQJob* d_jobs, const int* d_col_off, int njobs, int total_cols, int es,
                       cudaStream_t s) {
  if (njobs <= 0 || total_cols <= 0) return 0;
  if (!valid_es(es)) return (int)cudaErrorInvalidValue;
  const int grid = (total_cols + kW - 1) / kW;
  if (es == 16) formq_kernel<double2><<<grid, kT, 0, s>>>(d_jobs, d_col_off, njobs, total_cols);
  else formq_kernel<float2><<<grid, kT, 0, s>>>(d_jobs, d_col_off, njobs, total_cols);
  return (int)cudaGetLastError();
}
namespace {
template <typename C, int WM, int WN, int NS>
int launch_gemm_ns(const GemmBatch& g, int tk, cudaStream_t s) {
  static SmemLimit attr;
  if (const int e = smem_limit(gemm_kernel<C, WM, WN, NS>, attr)) return e;
  const size_t smem = sizeof(C) * NS * (size_t)(gemm_area(8 * WM, tk) + gemm_area(8 * WN, tk));
  GemmInline<NS> inl;
  dim3 grid(g.ntiles);
  if (!g.d) {
    memcpy(inl.b, g.one, sizeof(GemmOne) * g.none);
    grid = dim3(g.ntiles, g.none);  // ntiles: the most tiles of one product
  }
  return launch_chain(gemm_kernel<C, WM, WN, NS>, grid, 32 * WM * WN * (NS == 1 ? 1 : 2), smem, s, g.d, g.terms, g.tiles,
                      tk, inl);
}
template <typename C, int WM, int WN>
int launch_gemm(const GemmBatch& g, cudaStream_t s) {
  // every product one chunk: one buffer, so that many CTAs share an SM
  if (!g.d || (g.tmax <= 1 && g.kmax <= kGemmTK1))
    return launch_gemm_ns<C, WM, WN, 1>(g, std::max(4, (g.kmax + 3) & ~3), s);
  const int tk = std::max(4, std::min(kGemmTK, (g.kmax + 3) & ~3));
  // few CTAs: four buffers hide more of the load latency; many: three, for more CTAs an SM
  if (g.ntiles <= 2 * 148 && 8 * WM < 32) return launch_gemm_ns<C, WM, WN, 4>(g, tk, s);
  return launch_gemm_ns<C, WM, WN, 3>(g, tk, s);
}
}  // namespace
void aifmm_gemm_tile(int shape, int* tm, int* tn) {
  *tm = shape == 16 ? 16 : 32;
  *tn = shape;
}
bool aifmm_gemm_inline(int nproducts, int kmax, int tmax) {
  return nproducts <= kGemmInline && kmax <= kGemmTK1 && tmax <= 1;
}
int aifmm_launch_gemm(const GemmBatch& g, int shape, cudaStream_t s, int es) {
  if (g.ntiles <= 0) return 0;
  if (!valid_es(es) || (!g.d && !aifmm_gemm_inline(g.none, g.kmax, g.tmax))) return (int)cudaErrorInvalidValue;
  switch (shape) {
#define AIFMM_GEMM_CASE(S, WM, WN) \
    case S: return es == 16 ? launch_gemm<double2, WM, WN>(g, s) : launch_gemm<float2, WM, WN>(g, s);
    AIFMM_GEMM_CASE(8, 4, 1) AIFMM_GEMM_CASE(16, 2, 2) AIFMM_GEMM_CASE(32, 4, 4)
#undef AIFMM_GEMM_CASE
  }
  return (int)cudaErrorInvalidValue;
}
int aifmm_geam_inline_max() { return kGeamInline; }
int aifmm_launch_geam(const GeamDesc* d, const GeamDesc* h, int nd, int max_elems, cudaStream_t s) {
  if (nd <= 0 || max_elems <= 0) return 0;
  if (!d && nd > kGeamInline) return (int)cudaErrorInvalidValue;
  GeamInline inl;
  if (!d) memcpy(inl.b, h, sizeof(GeamDesc) * nd);
  // four elements a thread; few blocks: one each, so that a small copy is one round of loads
  const int per = nd > 1024 ? 1024 : 256;
  const int gx = std::min(std::max(1, (max_elems + per - 1) / per), 148 * 4);
  return launch_chain(geam_kernel, dim3(gx, std::min(nd, 65535)), 256, 0, s, d, nd, inl);
}
int aifmm_launch_equilibrate(const EquilDesc* d, int nd, cudaStream_t s) {
  if (nd <= 0) return 0;
  equilibrate_kernel<<<nd, kT, 0, s>>>(d);
  return (int)cudaGetLastError();
}
int aifmm_norm_inline_max() { return kNormInline; }
int aifmm_launch_norms(const NormDesc* d, const NormDesc* h, int nd, cudaStream_t s) {
  if (nd <= 0) return 0;
  if (!d && nd > kNormInline) return (int)cudaErrorInvalidValue;
  NormInline inl;
  if (!d) memcpy(inl.b, h, sizeof(NormDesc) * nd);
  return launch_chain(norm_kernel, dim3(nd), kT, 0, s, d, inl);
}
int aifmm_launch_skel_lu(const SkelLUJob* d, int nd, const EntryCtx& ctx, cudaStream_t s) {
  if (nd <= 0) return 0;
  skel_lu_kernel<<<nd, kT, 0, s>>>(d, ctx);
  return (int)cudaGetLastError();
}
