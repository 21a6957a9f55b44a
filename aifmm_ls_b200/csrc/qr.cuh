// qr.cuh -- column-pivoted QR of the elimination's small blocks, for the
// factorisation kernels (k_qr.cu) and the fused recompression (k_compress.cu).
// Semantics of the factorisation: see k_dense.cu.
//
// Two kernels share the arithmetic, operation for operation, so that a block's
// factors do not depend on which one takes it:
//  * qr_reg: the columns live in registers (blocks up to 144 rows; limits at
//    qr_class below);
//  * qr_smem: the matrix in shared memory (what the registers do not hold).
#pragma once
#include <algorithm>
#include "dense.cuh"

namespace {

constexpr int kQrGroups = kT / 4;

// ---------------------------------------------------------------- register QR
// Four lanes own one column (rows p, p + 4, ... in lane p), every column of the
// block at once: 4 n threads.  A pivot step k:
//   1. every warp takes the largest (squared, downdated) norm from shared memory;
//      a group whose norm's high word is the only one there owns the pivot.  Where
//      two come within one unit of the high word, the positions and norms go
//      through shared memory and the tie rule of qr_smem_body decides;
//   2. the owner turns its column into the reflector, in registers and in V, while
//      the others take the square roots of their norms;
//   3. barrier; every other group applies it to its column, downdates the norm and
//      prepares the next step: its element of row k + 1 and the sum of squares below;
//   4. barrier.
// What bounds it: the chain of a step -- the norm reduction, square root and
// division of the reflector, the columns' dot products, the square root of the
// downdate -- not FP64 throughput: about 2,500 cycles a step.  36 x 57 complex128:
// 94 us with the shared-memory kernel, 49 us here; 64 x 64: 180 and 101 us; 90 x 90: 406
// and 255 us.  Finished columns stay in registers until the
// end; rows above 4 I0 are finished in phase I0 and cost nothing there.
// Sums run in the order of qr_smem_body, so that a block's factors do not depend on
// the kernel that takes it: lane p adds its rows with i = row / 4 even and odd in two
// partial sums; the reflector's sum of squares is the tree that 32 lanes form over
// the rows k + 1 + l (l mod 32), whose levels 16, 8 and 4 pair rows of one lane.
__host__ __device__ constexpr int qr_threads(int rpl) {
  return rpl <= 9 ? 512 : rpl <= 16 ? 384 : rpl <= 24 ? 384 : 256;
}
__host__ __device__ constexpr int qr_phase_rows(int rpl) { return (rpl + 2) / 3; }

template <typename C>
struct RegQr {
  int m, n, size, lane, p, g;
  C* V;                // the reflector below row k
  unsigned* hi2;       // 2 x n: high words of the squared norms, by step parity; 0 = finished
  double* snu;         // n: norms, for the tie rule
  int* spos;           // n: positions, for the tie rule (-1: finished)
  double* srd;         // size: |R_kk|
  C* s_tau;
  int* s_pos;          // position of the pivot column before the swap
  int* s_nzp;
  double thr_helper, downdate_thr;
  // this group's column
  double tt, nd, z;    // squared norm, norm at the last recompute, sum of squares below row k
  C a, tau;            // element of row k; the reflector's coefficient once finished
  int pos;
  bool done, fresh;    // fresh: tt was recomputed, nd = sqrt(tt) is due
};

// the sum of squares of this column's rows > k0 in the order of 32 lanes over rows k0 + 1 + l
template <typename C, int RPL, int I0>
__device__ __forceinline__ double qr_reg_tail(const C (&col)[RPL], int k0, int p, int nfree, unsigned full) {
  double s[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = I0; i < RPL; ++i)
    if (i >= nfree || p + 4 * i > k0) s[i & 7] += cabs2_p(col[i]);
  double z = ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
  z += __shfl_xor_sync(full, z, 2);
  z += __shfl_xor_sync(full, z, 1);
  return z;
}

template <typename C, int RPL, int NQ, int I0>
__device__ __forceinline__ void qr_reg_phase(RegQr<C>& S, C (&col)[RPL]) {
  constexpr int I1 = I0 + qr_phase_rows(RPL) < RPL ? I0 + qr_phase_rows(RPL) : RPL;
  constexpr int I2 = I1 + 1 < RPL ? I1 + 1 : RPL;  // row k + 1 may be the next phase's first
  const unsigned full = 0xffffffffu;
  const int m = S.m, n = S.n, lane = S.lane, p = S.p;
  const int kend = min(4 * I1, S.size);
  C* const V = S.V;
  for (int k = 4 * I0; k < kend; ++k) {
    // 1. pivot
    const unsigned* hi = S.hi2 + (k & 1) * n;
    unsigned h[NQ], mh = 0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      h[q] = 0;
      if (32 * q < n && lane + 32 * q < n) h[q] = hi[lane + 32 * q];
      mh = max(mh, h[q]);
    }
    mh = __reduce_max_sync(full, mh);
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < NQ; ++q) cnt += h[q] + 1 >= mh;
    const unsigned one = __ballot_sync(full, cnt > 0), more = __ballot_sync(full, cnt > 1);
    bool owner;
    // not a number (high word above infinity's), zero or no clear maximum
    if (mh < 2 || mh > 0x7ff00000u || more != 0 || (one & (one - 1)) != 0) {
      if (p == 0 && S.g < n) { S.snu[S.g] = sqrt(S.tt); S.spos[S.g] = S.done ? -1 : S.pos; }
      __syncthreads();
      unsigned uh = 0, ul = 0;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int s = lane + 32 * q;
        if (s < n && S.spos[s] >= 0) {
          const unsigned vh = (unsigned)__double2hiint(S.snu[s]), vl = (unsigned)__double2loint(S.snu[s]);
          if (vh > uh || (vh == uh && vl > ul)) { uh = vh; ul = vl; }
        }
      }
      const unsigned xh = __reduce_max_sync(full, uh);
      const unsigned xl = __reduce_max_sync(full, uh == xh ? ul : 0u);
      const double cut = __hiloint2double((int)xh, (int)xl) * (1.0 - kPivotTie);
      unsigned key = 0xffffffffu, low = 0xffffffffu;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int s = lane + 32 * q;
        if (s < n && S.spos[s] >= 0) {
          const unsigned c = (unsigned)S.spos[s] * 1024u + (unsigned)s;
          low = min(low, c);
          if (S.snu[s] >= cut) key = min(key, c);
        }
      }
      key = __reduce_min_sync(full, key);
      if (key == 0xffffffffu) key = __reduce_min_sync(full, low);  // norms that are not numbers: no swap
      owner = S.g == (int)(key & 1023u);
    } else {
      owner = !S.done && (unsigned)__double2hiint(S.tt) + 1 >= mh;
    }
    // 2. the owner's reflector, rows k..m-1; the others' norms
    const double2 c0 = c2d(S.a);
    const double root = sqrt(owner ? cabs2_p(c0) + S.z : S.tt);
    double rkk = 0.0;
    if (owner) {
      double beta;
      C t;
      double2 rden;
      const bool null = S.z <= DBL_MIN && c0.y * c0.y <= DBL_MIN;
      if (null) {
        beta = c0.x;
        t = cplx<C>::mk(0.0, 0.0);
        rden = make_double2(0.0, 0.0);
      } else {
        beta = root;
        if (c0.x >= 0.0) beta = -beta;
        const double2 den = make_double2(c0.x - beta, c0.y);
        const double dd = cabs2_p(den);
        const double prod = beta * dd;
        double ib, idd;  // 1/beta, 1/|den|^2
        if (fabs(prod) > 1e-290 && fabs(prod) < 1e290) {
          const double q = 1.0 / prod;
          ib = dd * q;
          idd = beta * q;
        } else {
          ib = 1.0 / beta;
          idd = 1.0 / dd;
        }
        t = cplx<C>::from(make_double2((beta - c0.x) * ib, c0.y * ib));  // conj((beta - a_kk) / beta)
        rden = make_double2(den.x * idd, -den.y * idd);                  // 1 / (a_kk - beta)
      }
#pragma unroll
      for (int i = I0; i < RPL; ++i)
        if ((unsigned)(p + 4 * i - k - 1) < (unsigned)(m - k - 1)) {
          col[i] = null ? cplx<C>::mk(0.0, 0.0) : cplx<C>::from(cmul_p(c2d(col[i]), rden));
          V[p + 4 * i] = col[i];
        }
#pragma unroll
      for (int i = I0; i < I1; ++i)
        if (p + 4 * i == k) col[i] = cplx<C>::mk(beta, 0.0);
      if (p == 0) {
        *S.s_tau = t;
        *S.s_pos = S.pos;
      }
      S.tau = t;
      S.pos = k;
      S.done = true;
      rkk = fabs(beta);
    }
    __syncthreads();
    if (owner && p == 0) {
      S.srd[k] = rkk;
      // exactly nonzero pivots; the norm itself only near the threshold
      const double lim = S.thr_helper * (double)(m - k);
      if (!(S.tt > 2.0 * lim) && *S.s_nzp == S.size) {
        const double nub = sqrt(S.tt);
        if (nub * nub < lim) *S.s_nzp = k;
      }
    }
    // 3. G = I - t v v^H on the columns at positions > k; norm downdates.  The lanes of
    //    finished columns run along with a zero update, so that a warp never splits and
    //    its shuffles name all lanes; a warp of finished columns skips the step.
    unsigned hnext = 0;
    if (!__all_sync(full, S.done)) {
      const bool on = !S.done;
      const double nu = root;
      if (on && S.fresh) S.nd = nu;
      S.fresh = false;
      const C t = *S.s_tau;
      if (on && S.pos == k) S.pos = *S.s_pos;
      C d0 = cplx<C>::mk(0.0, 0.0), d1 = cplx<C>::mk(0.0, 0.0);
#pragma unroll
      for (int i = I0; i < RPL; ++i)
        if (i >= I1 || p + 4 * i > k) {
          if (i & 1) d1 = cfmac(V[p + 4 * i], col[i], d1);
          else d0 = cfmac(V[p + 4 * i], col[i], d0);
        }
      C d = cadd(d0, d1);
      d.x += __shfl_xor_sync(full, d.x, 1); d.y += __shfl_xor_sync(full, d.y, 1);
      d.x += __shfl_xor_sync(full, d.x, 2); d.y += __shfl_xor_sync(full, d.y, 2);
      C tw = cmul_t(t, cadd(S.a, d));
      const C rkj = csub(S.a, tw);
      if (!on) tw = cplx<C>::mk(0.0, 0.0);
      if (RPL > 16) asm volatile("" ::: "memory");  // read v again rather than keep it in registers
#pragma unroll
      for (int i = I0; i < RPL; ++i)
        if (i >= I1 || p + 4 * i > k) col[i] = csub(col[i], cmul_p(V[p + 4 * i], tw));
#pragma unroll
      for (int i = I0; i < I1; ++i)
        if (on && p + 4 * i == k) col[i] = rkj;
      // the next step's element and sum of squares
      C an = cplx<C>::mk(0.0, 0.0);
#pragma unroll
      for (int i = I0; i < I2; ++i)
        if (p + 4 * i == k + 1) an = col[i];
      const int src = (lane & ~3) | ((k + 1) & 3);
      S.a.x = __shfl_sync(full, an.x, src);
      S.a.y = __shfl_sync(full, an.y, src);
      S.z = qr_reg_tail<C, RPL, I0>(col, k + 1, p, I2, full);
      const double ar = sqrt(cabs2_p(rkj));
      double tt = (nu - ar) * (nu + ar);
      if (tt < 0.0) tt = 0.0;
      const bool again = on && nu != 0.0 && tt <= S.downdate_thr * (S.nd * S.nd);
      if (__any_sync(full, again)) {
        double q = 0.0;
#pragma unroll
        for (int i = I0; i < RPL; ++i)
          if (i >= I1 || p + 4 * i > k) q += cabs2_p(col[i]);
        q += __shfl_xor_sync(full, q, 1);
        q += __shfl_xor_sync(full, q, 2);
        if (again) { tt = q; S.fresh = true; }
      }
      if (on && nu != 0.0) S.tt = tt;
      if (on) hnext = (unsigned)__double2hiint(S.tt);
    }
    if (p == 0 && S.g < n) S.hi2[((k + 1) & 1) * n + S.g] = hnext;
    __syncthreads();
  }
  if constexpr (I1 < RPL) {
    if (S.size > 4 * I1) qr_reg_phase<C, RPL, NQ, I1>(S, col);
  }
}

// Shared memory of the body.
__host__ __device__ inline size_t qr_reg_smem_bytes(int rpl, int n, int size, int es) {
  return (size_t)es * (4 * rpl + 1) + sizeof(double) * ((size_t)n + size) + sizeof(int) * (3 * (size_t)n + 2) + 32;
}

// QR of the m x n block whose element (row, slot) is load(row, slot): finished
// column k to out + k ldo (columns that were never pivots too, if rest), tau and
// perm (may be nullptr) likewise; info[0] = nonzero pivots, info[1] = rank.
// Starts with a barrier after the loads, ends with one after the last write.
template <typename C, int RPL, typename Load>
__device__ __forceinline__ void qr_reg_body(int m, int n, Load load, C* out, int ldo, C* tau, int* perm, bool rest,
                                            double thr_, int* info, double* maxpiv_out, char* smem) {
  constexpr int NQ = (qr_threads(RPL) / 4 + 31) / 32;
  RegQr<C> S;
  S.m = m; S.n = n; S.size = min(m, n);
  const int tid = threadIdx.x;
  S.lane = tid & 31; S.p = tid & 3; S.g = tid >> 2;
  S.V = reinterpret_cast<C*>(smem);
  S.s_tau = S.V + 4 * RPL;
  S.snu = reinterpret_cast<double*>(smem + ((sizeof(C) * (4 * RPL + 1) + 15) & ~size_t(15)));
  S.srd = S.snu + n;
  S.hi2 = reinterpret_cast<unsigned*>(S.srd + S.size);
  S.spos = reinterpret_cast<int*>(S.hi2 + 2 * n);
  S.s_pos = S.spos + n;
  S.s_nzp = S.s_pos + 1;
  const bool mine = S.g < n;
  const unsigned full = 0xffffffffu;
  C col[RPL];
#pragma unroll
  for (int i = 0; i < RPL; ++i) {
    const int row = S.p + 4 * i;
    col[i] = mine && row < m ? load(row, S.g) : cplx<C>::mk(0.0, 0.0);
  }
  double q = 0.0;
#pragma unroll
  for (int i = 0; i < RPL; ++i)
    if (S.p + 4 * i < m) q += cabs2_p(col[i]);
  q += __shfl_xor_sync(full, q, 1);
  q += __shfl_xor_sync(full, q, 2);
  S.tt = q;
  S.nd = sqrt(q);
  S.fresh = false;
  S.done = !mine;
  S.pos = S.g;
  S.a.x = __shfl_sync(full, col[0].x, S.lane & ~3);
  S.a.y = __shfl_sync(full, col[0].y, S.lane & ~3);
  S.z = qr_reg_tail<C, RPL, 0>(col, 0, S.p, 1, full);
  S.tau = cplx<C>::mk(0.0, 0.0);
  if (mine && S.p == 0) { S.snu[S.g] = S.nd; S.hi2[S.g] = (unsigned)__double2hiint(q); }
  // rows m .. 4 RPL - 1 of V are read as zeros
  for (int i = m + tid; i < 4 * RPL; i += blockDim.x) S.V[i] = cplx<C>::mk(0.0, 0.0);
  if (tid == 0) *S.s_nzp = S.size;
  __syncthreads();
  double maxnorm = 0.0;
#pragma unroll
  for (int u = 0; u < NQ; ++u)
    if (S.lane + 32 * u < n) maxnorm = fmax(maxnorm, S.snu[S.lane + 32 * u]);
  for (int o = 16; o > 0; o >>= 1) maxnorm = fmax(maxnorm, __shfl_xor_sync(full, maxnorm, o));
  const double eps = rl<typename cplx<C>::R>::eps;  // the precision of the data
  S.thr_helper = m > 0 ? (maxnorm * eps) * (maxnorm * eps) / m : 0.0;
  S.downdate_thr = sqrt(eps);
  __syncthreads();  // snu is written again by the tie rule
  if (S.size > 0) qr_reg_phase<C, RPL, NQ, 0>(S, col);
  // columns that were never pivots (positions >= size) only if asked for
  if (mine && (S.done || rest)) {
#pragma unroll
    for (int i = 0; i < RPL; ++i)
      if (S.p + 4 * i < m) out[S.p + 4 * i + (size_t)S.pos * ldo] = col[i];
    if (S.p == 0) {
      if (S.done) tau[S.pos] = S.tau;
      if (perm) perm[S.pos] = S.g;
    }
  }
  if (tid == 0) {
    double maxpivot = 0.0;
    for (int i = 0; i < S.size; ++i) maxpivot = fmax(maxpivot, S.srd[i]);
    const double thr = thr_ > 0.0 ? thr_ : (double)S.size * eps;
    const double pre = fabs(maxpivot) * thr;
    const int nzp = *S.s_nzp;
    int rk = 0;
    for (int i = 0; i < nzp; ++i) rk += (S.srd[i] > pre);
    info[0] = nzp;
    info[1] = rk;
    if (maxpiv_out) maxpiv_out[0] = maxpivot;
  }
  __syncthreads();
}

// Jobs whose matrix fits in shared memory, one barrier per pivot step.
// The matrix sits in shared memory by original column ("slot"); a column swap
// only exchanges the positions that two slots carry.  Each pivot step:
//   1. every warp selects the pivot from the shared norms/positions and builds
//      the reflector from the pivot column into its own buffer (all warps get the
//      same bits: same data, same reduction order), so no warp waits for another;
//   2. warp (k mod warps) writes the finished pivot column -- R above, beta on,
//      the reflector below the diagonal -- straight to global memory;
//   3. the four lanes of a group apply the reflector to each column the group
//      owns (slots g, g + 64, ...; rows interleaved over the lanes) and downdate
//      its norm;
//   4. one barrier.
// Norms and positions are double-buffered by step parity, so a warp running
// ahead never changes what a slower warp is still scanning.  Columns left at
// positions >= min(m, n) are written out at the end.
// Arithmetic: pivot ties as in qr_factor_kernel (kPivotTie); the reflector scalars tau and
// 1/(a_kk - beta) come from one division; the norm downdate of LAPACK Working
// Note 176 is evaluated without divisions -- with T = (nu - |r|)(nu + |r|) (the
// LAWN quantity (1 - (|r|/nu)^2) times nu^2), the column is recomputed when
// T <= sqrt(eps) nd^2 and otherwise nu becomes sqrt(T).
__host__ __device__ __forceinline__ int qr_smem_ld(int m) { return m + ((12 - (m & 7)) & 7); }  // ld = 4 (mod 8)

template <typename C>
__device__ void qr_smem_body(const QRJob& J, C* qsm) {
  const int m = J.m, n = J.n, size = min(m, n);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, p = tid & 3, g = tid >> 2;
  const int ld = qr_smem_ld(m);
  const unsigned full = 0xffffffffu, gm = 0xfu << (lane & ~3);
  C* A = qsm;                                                    // ld x n, by slot
  C* V = A + (size_t)ld * n;                                     // kW x m: each warp's reflector
  double* snu2 = reinterpret_cast<double*>(V + (size_t)kW * m);  // 2 x n: norms, by step parity
  double* snd = snu2 + 2 * n;                                    // n: norms at the last recompute
  double* srd = snd + n;                                         // size: |R_kk|
  int* spos2 = reinterpret_cast<int*>(srd + size);               // 2 x n: positions, by step parity
  const C* Ja = static_cast<const C*>(J.a);
  C* Jout = static_cast<C*>(J.a);
  C* Jtau = static_cast<C*>(J.tau);
  for (int e = tid; e < m * n; e += kT) {
    const int i = e % m, j = e / m;
    A[i + (size_t)j * ld] = Ja[i + (size_t)j * J.lda];
  }
  __syncthreads();
  for (int s = g; s < n; s += kQrGroups) {
    const C* col = A + (size_t)s * ld;
    double q = 0.0;
    for (int i = p; i < m; i += 4) q += cabs2_p(col[i]);
    q += __shfl_xor_sync(gm, q, 1);
    q += __shfl_xor_sync(gm, q, 2);
    if (p == 0) { snu2[s] = snd[s] = sqrt(q); spos2[s] = s; }
  }
  __syncthreads();
  const int nscan = (n + 31) >> 5;
  double maxnorm = 0.0;
  for (int q = 0; q < nscan; ++q) { const int s = lane + 32 * q; if (s < n) maxnorm = fmax(maxnorm, snu2[s]); }
  for (int o = 16; o > 0; o >>= 1) maxnorm = fmax(maxnorm, __shfl_xor_sync(full, maxnorm, o));
  const double eps = rl<typename cplx<C>::R>::eps;  // the precision of the data
  const double thr_helper = m > 0 ? (maxnorm * eps) * (maxnorm * eps) / m : 0.0;
  const double downdate_thr = sqrt(eps);
  C* vw = V + (size_t)w * m;
  int nzp = size;
  double maxpivot = 0.0;
  for (int k = 0; k < size; ++k) {
    const double* snu = snu2 + (k & 1) * n;
    const int* spos = spos2 + (k & 1) * n;
    double* snu_n = snu2 + ((k + 1) & 1) * n;
    int* spos_n = spos2 + ((k + 1) & 1) * n;
    // 1. pivot: largest norm at positions >= k, the first position within the
    //    tie tolerance.  Norms are non-negative: their bit patterns order like
    //    their values, so the maximum is two unsigned warp reductions.
    unsigned hi = 0, lo = 0;
    for (int q = 0; q < nscan; ++q) {
      const int s = lane + 32 * q;
      if (s < n && spos[s] >= k) {
        const double v = snu[s];
        const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
        if (h > hi || (h == hi && l > lo)) { hi = h; lo = l; }
      }
    }
    const unsigned mh = __reduce_max_sync(full, hi);
    const unsigned ml = __reduce_max_sync(full, hi == mh ? lo : 0u);
    const double cut = __hiloint2double((int)mh, (int)ml) * (1.0 - kPivotTie);
    unsigned key = 0xffffffffu;
    for (int q = 0; q < nscan; ++q) {
      const int s = lane + 32 * q;
      if (s < n) {
        const int ps = spos[s];
        if (ps >= k && snu[s] >= cut) key = min(key, (unsigned)ps * 1024u + (unsigned)s);
      }
    }
    key = __reduce_min_sync(full, key);
    if (key == 0xffffffffu) {  // norms that are not numbers: no swap, as in qr_reg_phase
      for (int q = 0; q < nscan; ++q) {
        const int s = lane + 32 * q;
        if (s < n && spos[s] >= k) key = min(key, (unsigned)spos[s] * 1024u + (unsigned)s);
      }
      key = __reduce_min_sync(full, key);
    }
    const int big = (int)(key >> 10), bslot = (int)(key & 1023u);
    const double nub = snu[bslot];
    if (nzp == size && nub * nub < thr_helper * (double)(m - k)) nzp = k;
    //    reflector for the pivot column, rows k..m-1
    const C* pc = A + (size_t)bslot * ld;
    double tail = 0.0;
    for (int i = k + 1 + lane; i < m; i += 32) tail += cabs2_p(pc[i]);
    for (int o = 16; o > 0; o >>= 1) tail += __shfl_xor_sync(full, tail, o);
    const double2 c0 = c2d(pc[k]);
    double beta;
    C t;
    if (tail <= DBL_MIN && c0.y * c0.y <= DBL_MIN) {
      beta = c0.x;
      t = cplx<C>::mk(0.0, 0.0);
      for (int i = k + 1 + lane; i < m; i += 32) vw[i] = cplx<C>::mk(0.0, 0.0);
    } else {
      beta = sqrt(cabs2_p(c0) + tail);
      if (c0.x >= 0.0) beta = -beta;
      const double2 den = make_double2(c0.x - beta, c0.y);
      const double dd = cabs2_p(den);
      const double prod = beta * dd;
      double ib, idd;  // 1/beta, 1/|den|^2
      if (fabs(prod) > 1e-290 && fabs(prod) < 1e290) {
        const double q = 1.0 / prod;
        ib = dd * q;
        idd = beta * q;
      } else {
        ib = 1.0 / beta;
        idd = 1.0 / dd;
      }
      t = cplx<C>::from(make_double2((beta - c0.x) * ib, c0.y * ib));  // conj((beta - a_kk) / beta)
      const double2 rden = make_double2(den.x * idd, -den.y * idd);    // 1 / (a_kk - beta)
      for (int i = k + 1 + lane; i < m; i += 32) vw[i] = cplx<C>::from(cmul_p(c2d(pc[i]), rden));
    }
    maxpivot = fmax(maxpivot, fabs(beta));
    __syncwarp();
    // 2. the finished pivot column goes to position k
    if (w == (k & (kW - 1))) {
      C* out = Jout + (size_t)k * J.lda;
      for (int i = lane; i < m; i += 32) out[i] = i < k ? pc[i] : (i == k ? cplx<C>::mk(beta, 0.0) : vw[i]);
      if (lane == 0) { Jtau[k] = t; J.perm[k] = bslot; srd[k] = fabs(beta); }
    }
    // 3. G = I - t v v^H on the columns at positions > k; norm downdates
    for (int s = g; s < n; s += kQrGroups) {
      int ps = spos[s];
      if (ps == big) ps = k;
      else if (ps == k) ps = big;
      if (ps > k) {
        C* col = A + (size_t)s * ld;
        const int i0 = k + 1 + ((p - (k + 1)) & 3);  // this lane's first row below k
        C d0 = cplx<C>::mk(0.0, 0.0), d1 = cplx<C>::mk(0.0, 0.0);
        int i = i0;
        for (; i + 4 < m; i += 8) { d0 = cfmac(vw[i], col[i], d0); d1 = cfmac(vw[i + 4], col[i + 4], d1); }
        if (i < m) d0 = cfmac(vw[i], col[i], d0);
        C d = cadd(d0, d1);
        d.x += __shfl_xor_sync(gm, d.x, 1); d.y += __shfl_xor_sync(gm, d.y, 1);
        d.x += __shfl_xor_sync(gm, d.x, 2); d.y += __shfl_xor_sync(gm, d.y, 2);
        const C akj = col[k];
        const C tw = cmul_t(t, cadd(akj, d));
        for (int r = i0; r < m; r += 4) col[r] = csub(col[r], cmul_p(vw[r], tw));
        const C rkj = csub(akj, tw);
        __syncwarp(gm);
        if (p == 0) col[k] = rkj;
        double nu = snu[s], nd = snd[s];
        if (nu != 0.0) {
          const double ar = sqrt(cabs2_p(rkj));
          double tt = (nu - ar) * (nu + ar);
          if (tt < 0.0) tt = 0.0;
          if (tt <= downdate_thr * (nd * nd)) {
            double q = 0.0;
            for (int r = i0; r < m; r += 4) q += cabs2_p(col[r]);
            q += __shfl_xor_sync(gm, q, 1);
            q += __shfl_xor_sync(gm, q, 2);
            nd = sqrt(q);
            nu = nd;
          } else {
            nu = sqrt(tt);
          }
        }
        if (p == 0) { snu_n[s] = nu; snd[s] = nd; }
      }
      if (p == 0) spos_n[s] = ps;
    }
    __syncthreads();
  }
  // 4. columns that were never pivots (positions >= size)
  const int* spos = spos2 + (size & 1) * n;
  for (int s = g; s < n; s += kQrGroups) {
    const int ps = spos[s];
    if (ps >= size) {
      const C* col = A + (size_t)s * ld;
      C* out = Jout + (size_t)ps * J.lda;
      for (int i = p; i < m; i += 4) out[i] = col[i];
      if (p == 0) J.perm[ps] = s;
    }
  }
  if (tid == 0) {
    const double thr = J.thr > 0.0 ? J.thr : (double)size * eps;
    const double pre = fabs(maxpivot) * thr;
    int rk = 0;
    for (int i = 0; i < nzp; ++i) rk += (srd[i] > pre);
    J.info[0] = nzp;
    J.info[1] = rk;
    if (J.maxpiv) J.maxpiv[0] = maxpivot;
  }
}

// The register kernels by rows per lane; a block takes the smallest that holds its
// rows, if its columns fit that kernel's threads (qr_threads: 65,536 registers
// divided by what a column of that many rows needs).  -1: the shared-memory kernel.
constexpr int kRpl[] = {5, 9, 16, 24, 36};
constexpr int kClasses = sizeof kRpl / sizeof kRpl[0];
int qr_class(int m, int n) {
  for (int c = 0; c < kClasses; ++c)
    if (m <= 4 * kRpl[c]) return 4 * n <= qr_threads(kRpl[c]) ? c : -1;
  return -1;
}
int threads_for(int n) { return std::max(32, (4 * n + 31) / 32 * 32); }

}  // namespace
