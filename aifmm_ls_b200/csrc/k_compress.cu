// k_compress.cu -- one direction of compress_P2P (FMM2DTree_find_error.hpp:1532-1559)
// per CTA, on the register QR or, for blocks that it does not hold, on the
// shared-memory QR (qr.cuh).
#include <cstring>

#include "qr.cuh"

namespace {

// ---------------------------------------------------------------- fused compression
// CTA-wide building blocks on global-memory operands (written earlier by the
// same CTA; a __syncthreads separates producer and consumer).

// C (m x n, ldc) = alpha op(A) op(B) + beta C; op 1 = conjugate transpose.
// Accumulation over k in increasing order, as gemm_kernel.
template <typename C>
__device__ void cta_gemm(C* Cm, int ldc, int m, int n, int k, const C* A, int lda, int opA,
                         const C* B, int ldb, int opB, double2 alpha_, double2 beta_) {
  const bool zero_beta = beta_.x == 0.0 && beta_.y == 0.0;
  const C alpha = cplx<C>::from(alpha_), beta = cplx<C>::from(beta_);
  for (int o = threadIdx.x; o < m * n; o += kT) {
    const int i = o % m, jj = o / m;
    C acc = cplx<C>::mk(0.0, 0.0);
#pragma unroll 4
    for (int kk = 0; kk < k; ++kk) {
      const C a = opA ? cconj(A[kk + (size_t)i * lda]) : A[i + (size_t)kk * lda];
      const C b = opB ? cconj(B[jj + (size_t)kk * ldb]) : B[kk + (size_t)jj * ldb];
      acc = cfma(a, b, acc);
    }
    C v = cmul(alpha, acc);
    if (!zero_beta) v = cadd(v, cmul(beta, Cm[i + (size_t)jj * ldc]));
    Cm[i + (size_t)jj * ldc] = v;
  }
}

size_t aifmm_formq_smem_bytes(int m, int size, int ncols, int es) {
  return (size_t)es * ((size_t)(m | 1) * size + size + (size_t)m * ncols);
}

// Q(:, 0:ncols) = householderQ() of an m x n factor (reflectors below the
// diagonal of qr, coefficients tau): column c is G_0^H ... G_min(c, size-1)^H e_c.
// The factor is staged in shared memory; the four lanes of a group build one
// column (rows interleaved), reducing the reflector dot products by shuffles.
template <typename C>
__device__ void cta_formq(const C* qr, int ldq, int m, int n, const C* tau, C* Q, int ldQ, int ncols, C* sm) {
  const int size = min(m, n), ldf = m | 1;
  const int tid = threadIdx.x, lane = tid & 31, p = tid & 3, g = tid >> 2;
  const unsigned gm = 0xfu << (lane & ~3);
  C* F = sm;
  C* ts = F + (size_t)ldf * size;
  C* Qs = ts + size;
  for (int e = tid; e < m * size; e += kT) {
    const int i = e % m, j = e / m;
    F[i + (size_t)j * ldf] = qr[i + (size_t)j * ldq];
  }
  for (int k = tid; k < size; k += kT) ts[k] = cconj(tau[k]);
  for (int e = tid; e < m * ncols; e += kT) {
    const int i = e % m, j = e / m;
    Qs[e] = cplx<C>::mk(i == j ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  for (int cc = g; cc < ncols; cc += kQrGroups) {
    C* q = Qs + (size_t)cc * m;
    for (int k = min(size - 1, cc); k >= 0; --k) {
      const C* v = F + (size_t)k * ldf;
      const int i0 = k + 1 + ((p - (k + 1)) & 3);
      C d = cplx<C>::mk(0.0, 0.0);
      for (int i = i0; i < m; i += 4) d = cfmac(v[i], q[i], d);
      d.x += __shfl_xor_sync(gm, d.x, 1); d.y += __shfl_xor_sync(gm, d.y, 1);
      d.x += __shfl_xor_sync(gm, d.x, 2); d.y += __shfl_xor_sync(gm, d.y, 2);
      const C qk = q[k];
      const C tw = cmul_p(ts[k], cadd(qk, d));
      for (int i = i0; i < m; i += 4) q[i] = csub(q[i], cmul_p(v[i], tw));
      __syncwarp(gm);
      if (p == 0) q[k] = csub(qk, tw);
      __syncwarp(gm);
    }
  }
  __syncthreads();
  for (int e = tid; e < m * ncols; e += kT) {
    const int i = e % m, j = e / m;
    Q[i + (size_t)j * ldQ] = Qs[e];
  }
}

template <typename C>
__global__ void __launch_bounds__(kT) compress_p2p_kernel(const CompressJob* __restrict__ jobs) {
  extern __shared__ double2 csm_raw[];
  C* csm = reinterpret_cast<C*>(csm_raw);
  const CompressJob J = jobs[blockIdx.x];
  const int m = J.m, rK = J.rK, c = J.c, rb = J.rb, n1 = rK + c;
  const int tid = threadIdx.x;
  const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);
  const C* L2P = static_cast<const C*>(J.L2P);
  const C* Pkb = static_cast<const C*>(J.Pkb);
  const C* P2M = static_cast<const C*>(J.P2M);
  const C* M2L = static_cast<const C*>(J.M2L);
  C* Acol = static_cast<C*>(J.Acol);
  C* Arow = static_cast<C*>(J.Arow);
  C* tau = static_cast<C*>(J.tau);
  C* nL = static_cast<C*>(J.nL);
  C* nPt = static_cast<C*>(J.nPt);
  C* Rkp = static_cast<C*>(J.Rkp);
  C* Rk = static_cast<C*>(J.Rk);
  C* Rn = static_cast<C*>(J.Rn);
  C* Rnp = static_cast<C*>(J.Rnp);
  C* Tm = static_cast<C*>(J.Tm);
  C* M2Lo = static_cast<C*>(J.M2Lo);
  // [L2P_k | P2P_kb]
  for (int e = tid; e < m * n1; e += kT) {
    const int i = e % m, col = e / m;
    Acol[e] = col < rK ? L2P[i + (size_t)col * J.ldL] : Pkb[i + (size_t)(col - rK) * J.ldP];
  }
  __syncthreads();
  QRJob q{};
  q.a = Acol; q.lda = m; q.m = m; q.n = n1; q.tau = tau; q.perm = J.perm; q.info = J.info; q.thr = J.tol;
  qr_smem_body<C>(q, csm);
  __syncthreads();
  const int rc = J.info[1];
  const int ldc_ = max(rc, 1);
  cta_formq<C>(Acol, m, m, n1, tau, nL, m, rc, csm);
  __syncthreads();
  cta_gemm<C>(Rkp, ldc_, rc, c, m, nL, m, 1, Pkb, J.ldP, 0, one, zero);   // R' = nL^H P2P_kb
  cta_gemm<C>(Rk, ldc_, rc, rK, m, nL, m, 1, L2P, J.ldL, 0, one, zero);   // R = nL^H L2P_k
  __syncthreads();
  // [P2M_b^H | R'^H]
  const int n2 = rb + rc;
  for (int e = tid; e < c * n2; e += kT) {
    const int i = e % c, col = e / c;
    Arow[e] = col < rb ? cconj(P2M[col + (size_t)i * J.ldM]) : cconj(Rkp[(col - rb) + (size_t)i * ldc_]);
  }
  __syncthreads();
  q.a = Arow; q.lda = c; q.m = c; q.n = n2; q.info = J.info + 2;
  qr_smem_body<C>(q, csm);
  __syncthreads();
  const int rr = J.info[3];
  const int ldr_ = max(rr, 1);
  cta_formq<C>(Arow, c, c, n2, tau, nPt, c, rr, csm);
  __syncthreads();
  cta_gemm<C>(Rn, ldr_, rr, rb, c, nPt, c, 1, P2M, J.ldM, 1, one, zero);    // nPt^H P2M_b^H
  cta_gemm<C>(Rnp, ldr_, rr, rc, c, nPt, c, 1, Rkp, ldc_, 1, one, zero);    // nPt^H R'^H
  cta_gemm<C>(Tm, ldc_, rc, rb, rK, Rk, ldc_, 0, M2L, J.ldT, 0, one, zero);  // R M2L_kb
  __syncthreads();
  cta_gemm<C>(M2Lo, J.ldO, rc, rr, rb, Tm, ldc_, 0, Rn, ldr_, 1, one, zero);
  __syncthreads();
  for (int e = tid; e < rc * rr; e += kT) {
    const int i = e % rc, jj = e / rc;
    C* o = M2Lo + i + (size_t)jj * J.ldO;
    *o = cadd(cconj(Rnp[jj + (size_t)i * ldr_]), *o);
  }
  if (tid == 0) {  // may be mapped host memory
    J.ranks[0] = rc;
    J.ranks[1] = rr;
    __threadfence_system();
  }
}

// ---- the same with the register QR
// C (m x n, ldc) = op(A) op(B) [+ conj(D^T)]; op 1 = conjugate transpose.  A thread
// computes NU neighbouring outputs of one row, each over k in increasing order as in
// cta_gemm: one element of A serves all of them, and the elements of B are the same
// in most lanes of a warp.  (Loads of shared memory bound these products: with one
// load of A per output a 36 x 36 x 36 product took 10 us.)  Lanes run along the rows
// of C: an adjoint A has an odd leading dimension in shared memory.
template <typename C, int OPA, int OPB, bool ADD, int NU>
__device__ __forceinline__ void cta_gemm_n(C* Cm, int ldc, int m, int n, int k, const C* A, int lda, const C* B, int ldb,
                                           const C* D, int ldd) {
  const int tot = m * ((n + NU - 1) / NU);
  for (int o = threadIdx.x; o < tot; o += blockDim.x) {
    const int jg = o / m, i = o - jg * m, j0 = jg * NU;
    int jj[NU];
    C acc[NU];
#pragma unroll
    for (int u = 0; u < NU; ++u) {
      jj[u] = min(j0 + u, n - 1);
      acc[u] = cplx<C>::mk(0.0, 0.0);
    }
#pragma unroll 4
    for (int kk = 0; kk < k; ++kk) {
      const C a = OPA ? cconj(A[kk + i * lda]) : A[i + kk * lda];
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const C b = OPB ? cconj(B[jj[u] + kk * ldb]) : B[kk + jj[u] * ldb];
        acc[u] = cfma(a, b, acc[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < NU; ++u)
      if (j0 + u < n) {
        C v = acc[u];
        if (ADD) v = cadd(cconj(D[j0 + u + i * ldd]), v);
        Cm[i + (size_t)(j0 + u) * ldc] = v;
      }
  }
}
template <typename C, int OPA, int OPB, bool ADD = false>
__device__ __forceinline__ void cta_gemm_s(C* Cm, int ldc, int m, int n, int k, const C* A, int lda, const C* B, int ldb,
                                           const C* D = nullptr, int ldd = 0) {
  const int per = (m * n + blockDim.x - 1) / blockDim.x;
  if (per <= 2) cta_gemm_n<C, OPA, OPB, ADD, 2>(Cm, ldc, m, n, k, A, lda, B, ldb, D, ldd);
  else if (per <= 4) cta_gemm_n<C, OPA, OPB, ADD, 4>(Cm, ldc, m, n, k, A, lda, B, ldb, D, ldd);
  else cta_gemm_n<C, OPA, OPB, ADD, 6>(Cm, ldc, m, n, k, A, lda, B, ldb, D, ldd);
}

// One step range of formq: the reflectors k in [4 I0, 4 I1), downwards, on the
// group's column cc (nothing while k > cc).
// All lanes of a warp run along, those of columns without reflector k with a zero
// update, so that the shuffles name the whole warp.
template <typename C, int RPL, int I0>
__device__ __forceinline__ void formq_reg_phase(const C* F, int ldf, const C* tau, int m, int kmax, int cc, int p,
                                                int lane, C (&q)[RPL]) {
  constexpr int I1 = I0 + qr_phase_rows(RPL) < RPL ? I0 + qr_phase_rows(RPL) : RPL;
  if constexpr (I1 < RPL) formq_reg_phase<C, RPL, I1>(F, ldf, tau, m, kmax, cc, p, lane, q);
  const unsigned full = 0xffffffffu;
  for (int k = min(kmax, 4 * I1 - 1); k >= 4 * I0; --k) {
    const C* v = F + (size_t)k * ldf;
    const bool on = k <= cc;
    C qk = cplx<C>::mk(0.0, 0.0);
#pragma unroll
    for (int i = I0; i < I1; ++i)
      if (p + 4 * i == k) qk = q[i];
    const int src = (lane & ~3) | (k & 3);
    qk.x = __shfl_sync(full, qk.x, src);
    qk.y = __shfl_sync(full, qk.y, src);
    C d = cplx<C>::mk(0.0, 0.0);
#pragma unroll
    for (int i = I0; i < RPL; ++i)
      if ((unsigned)(p + 4 * i - k - 1) < (unsigned)(m - k - 1)) d = cfmac(v[p + 4 * i], q[i], d);
    d.x += __shfl_xor_sync(full, d.x, 1); d.y += __shfl_xor_sync(full, d.y, 1);
    d.x += __shfl_xor_sync(full, d.x, 2); d.y += __shfl_xor_sync(full, d.y, 2);
    C tw = cmul_p(cconj(tau[k]), cadd(qk, d));
    const C qn = csub(qk, tw);
    if (!on) tw = cplx<C>::mk(0.0, 0.0);
    if (RPL > 16) asm volatile("" ::: "memory");
#pragma unroll
    for (int i = I0; i < RPL; ++i)
      if ((unsigned)(p + 4 * i - k - 1) < (unsigned)(m - k - 1)) q[i] = csub(q[i], cmul_p(v[p + 4 * i], tw));
#pragma unroll
    for (int i = I0; i < I1; ++i)
      if (on && p + 4 * i == k) q[i] = qn;
  }
}

// Q(:, 0:ncols) of the factor in F (shared memory, ldf; its reflectors below the
// diagonal) to global memory (ld m) and, in place of the factor, to shared memory
// (ld ldf).  One group of four lanes per column, in registers.
template <typename C, int RPL>
__device__ __forceinline__ void cta_formq_reg(C* F, int ldf, const C* tau, int m, int size, int ncols, C* Q) {
  const int lane = threadIdx.x & 31, p = threadIdx.x & 3, cc = threadIdx.x >> 2;
  C q[RPL];
  if (cc - (lane >> 2) < ncols) {  // the same in a whole warp
#pragma unroll
    for (int i = 0; i < RPL; ++i) q[i] = cplx<C>::mk(p + 4 * i == cc ? 1.0 : 0.0, 0.0);
    formq_reg_phase<C, RPL, 0>(F, ldf, tau, m, min(size, ncols) - 1, cc, p, lane, q);
  }
  __syncthreads();
  if (cc < ncols) {
#pragma unroll
    for (int i = 0; i < RPL; ++i)
      if (p + 4 * i < m) {
        F[p + 4 * i + (size_t)cc * ldf] = q[i];
        Q[p + 4 * i + (size_t)cc * m] = q[i];
      }
  }
  __syncthreads();
}

constexpr int kCompressInline = 8;
using CompressInline = Inline<kCompressInline * sizeof(CompressJob)>;

// Where the operands of the compression live: the factor, the QR's own arrays, then
// the inputs and the intermediate products as far as shared memory goes; what does
// not fit stays in global memory (the kernel's code is the same: generic pointers).
constexpr size_t kCompressSmem = size_t(200) << 10;
struct CompressLayout {
  size_t body = 0, total = 0;
  size_t off[9];  // Pkb, L2P, P2M, M2L, R', R, Rn, Rn', T; 0: global memory
};
__host__ __device__ inline CompressLayout compress_layout(int rpl, int m, int rK, int c, int rb, int es) {
  CompressLayout L;
  const int n1 = rK + c, s1 = m < n1 ? m : n1, n2 = rb + s1, s2 = c < n2 ? c : n2;
  const size_t f1 = (size_t)(m | 1) * s1, f2 = (size_t)(c | 1) * s2;
  const int smax = s1 > s2 ? s1 : s2, nmax = n1 > n2 ? n1 : n2;
  L.body = ((size_t)es * ((f1 > f2 ? f1 : f2) + smax) + 15) & ~size_t(15);
  L.total = (L.body + qr_reg_smem_bytes(rpl, nmax, smax, es) + 31) & ~size_t(15);
  const size_t sz[9] = {(size_t)m * c,   (size_t)m * rK,  (size_t)rb * c,  (size_t)rK * rb, (size_t)s1 * c,
                        (size_t)s1 * rK, (size_t)s2 * rb, (size_t)s2 * s1, (size_t)s1 * rb};
  for (int i = 0; i < 9; ++i) {
    const size_t b = ((size_t)es * sz[i] + 15) & ~size_t(15);
    if (L.total + b <= kCompressSmem) { L.off[i] = L.total; L.total += b; }
    else L.off[i] = 0;
  }
  return L;
}

template <typename C>
__device__ __forceinline__ const C* stage(char* smem, size_t off, const void* src, int ld, int r, int n, int& ldo) {
  const C* g = static_cast<const C*>(src);
  ldo = ld;
  if (off == 0) return g;
  C* d = reinterpret_cast<C*>(smem + off);
  ldo = r > 0 ? r : 1;
  for (int e = threadIdx.x; e < r * n; e += blockDim.x) {
    const int j = e / r, i = e - j * r;
    d[e] = g[i + (size_t)j * ld];
  }
  return d;
}
template <typename C>
__device__ __forceinline__ C* place(char* smem, size_t off, void* g) {
  return off ? reinterpret_cast<C*>(smem + off) : static_cast<C*>(g);
}

template <typename C, int RPL>
__global__ void __launch_bounds__(qr_threads(RPL)) compress_reg_kernel(const CompressJob* __restrict__ jobs,
                                                                       const __grid_constant__ CompressInline inl) {
  extern __shared__ double2 csm_raw[];
  __shared__ int info[4];
  char* sm = reinterpret_cast<char*>(csm_raw);
  pdl_begin();
  const CompressJob J = jobs ? jobs[blockIdx.x] : reinterpret_cast<const CompressJob*>(inl.b)[blockIdx.x];
  pdl_wait();
  const int m = J.m, rK = J.rK, c = J.c, rb = J.rb, n1 = rK + c, s1 = min(m, n1);
  const CompressLayout L = compress_layout(RPL, m, rK, c, rb, (int)sizeof(C));
  int ldP, ldL, ldM, ldT;
  const C* Pkb = stage<C>(sm, L.off[0], J.Pkb, J.ldP, m, c, ldP);
  const C* L2P = stage<C>(sm, L.off[1], J.L2P, J.ldL, m, rK, ldL);
  const C* P2M = stage<C>(sm, L.off[2], J.P2M, J.ldM, rb, c, ldM);
  const C* M2L = stage<C>(sm, L.off[3], J.M2L, J.ldT, rK, rb, ldT);
  C* Rkp = place<C>(sm, L.off[4], J.Rkp);
  C* Rk = place<C>(sm, L.off[5], J.Rk);
  C* Rn = place<C>(sm, L.off[6], J.Rn);
  C* Rnp = place<C>(sm, L.off[7], J.Rnp);
  C* Tm = place<C>(sm, L.off[8], J.Tm);
  C* F = reinterpret_cast<C*>(sm);
  const int s2max = min(c, rb + s1);
  C* tau = F + max((m | 1) * s1, (c | 1) * s2max);
  char* body = sm + L.body;
  __syncthreads();
  // column QR of [L2P_k | P2P_kb]
  qr_reg_body<C, RPL>(
      m, n1, [&](int row, int slot) { return slot < rK ? L2P[row + slot * ldL] : Pkb[row + (slot - rK) * ldP]; }, F,
      m | 1, tau, nullptr, false, J.tol, info, nullptr, body);
  const int rc = info[1], ldc_ = max(rc, 1);
  cta_formq_reg<C, RPL>(F, m | 1, tau, m, s1, rc, static_cast<C*>(J.nL));
  cta_gemm_s<C, 1, 0>(Rkp, ldc_, rc, c, m, F, m | 1, Pkb, ldP);   // R' = nL^H P2P_kb
  cta_gemm_s<C, 1, 0>(Rk, ldc_, rc, rK, m, F, m | 1, L2P, ldL);   // R = nL^H L2P_k
  __syncthreads();
  // row QR of [P2M_b^H | R'^H]
  const int n2 = rb + rc;
  qr_reg_body<C, RPL>(
      c, n2,
      [&](int row, int slot) { return slot < rb ? cconj(P2M[slot + row * ldM]) : cconj(Rkp[(slot - rb) + row * ldc_]); },
      F, c | 1, tau, nullptr, false, J.tol, info + 2, nullptr, body);
  const int rr = info[3], ldr_ = max(rr, 1);
  cta_formq_reg<C, RPL>(F, c | 1, tau, c, min(c, n2), rr, static_cast<C*>(J.nPt));
  cta_gemm_s<C, 1, 1>(Rn, ldr_, rr, rb, c, F, c | 1, P2M, ldM);     // nPt^H P2M_b^H
  cta_gemm_s<C, 1, 1>(Rnp, ldr_, rr, rc, c, F, c | 1, Rkp, ldc_);   // nPt^H R'^H
  cta_gemm_s<C, 0, 0>(Tm, ldc_, rc, rb, rK, Rk, ldc_, M2L, ldT);    // R M2L_kb
  __syncthreads();
  cta_gemm_s<C, 0, 1, true>(static_cast<C*>(J.M2Lo), J.ldO, rc, rr, rb, Tm, ldc_, Rn, ldr_, Rnp, ldr_);
  if (threadIdx.x == 0) {  // may be mapped host memory
    J.ranks[0] = rc;
    J.ranks[1] = rr;
    __threadfence_system();
  }
}

template <typename C, int RPL>
int launch_compress_reg(const CompressJob* d_jobs, const CompressJob* h_jobs, int njobs, int n, size_t smem,
                        cudaStream_t s) {
  static SmemLimit attr;
  if (const int e = smem_limit(compress_reg_kernel<C, RPL>, attr)) return e;
  CompressInline inl;
  if (!d_jobs) memcpy(inl.b, h_jobs, sizeof(CompressJob) * njobs);
  return launch_chain(compress_reg_kernel<C, RPL>, dim3(njobs), threads_for(n), smem, s, d_jobs, inl);
}
}  // namespace

size_t aifmm_compress_smem_bytes(int m, int rK, int c, int rb, int es) {
  const int n1 = rK + c, s1 = std::min(m, n1), n2 = rb + s1, s2 = std::min(c, n2);
  if (m > 1024 || c > 1024) return 0;
  size_t b = std::max(aifmm_qr_smem_bytes(m, n1, es), aifmm_qr_smem_bytes(c, n2, es));
  b = std::max(b, aifmm_formq_smem_bytes(m, s1, s1, es));
  b = std::max(b, aifmm_formq_smem_bytes(c, s2, s2, es));
  return b <= (size_t(200) << 10) ? b : 0;
}
int aifmm_launch_compress_p2p(const CompressJob* d_jobs, int njobs, size_t smem, int es, cudaStream_t s) {
  if (njobs <= 0) return 0;
  if (!valid_es(es)) return (int)cudaErrorInvalidValue;
  static SmemLimit attr[2];
  if (es == 16) {
    if (const int e = smem_limit(compress_p2p_kernel<double2>, attr[0])) return e;
    compress_p2p_kernel<double2><<<njobs, kT, smem, s>>>(d_jobs);
  } else {
    if (const int e = smem_limit(compress_p2p_kernel<float2>, attr[1])) return e;
    compress_p2p_kernel<float2><<<njobs, kT, smem, s>>>(d_jobs);
  }
  return (int)cudaGetLastError();
}

// The class of the register kernel that takes both factorisations of a compression
// with these sizes, or -1.
int aifmm_compress_class(int m, int rK, int c, int rb, int es) {
  const int n1 = rK + c, s1 = std::min(m, n1), n2 = rb + s1;
  const int cls = qr_class(std::max(m, c), std::max(n1, n2));
  if (cls >= 0 && compress_layout(kRpl[cls], m, rK, c, rb, es).total > kCompressSmem) return -1;
  return cls;
}
// whether a class's kernel takes ncol columns
bool aifmm_compress_class_holds(int cls, int ncol) { return cls >= 0 && 4 * ncol <= qr_threads(kRpl[cls]); }
size_t aifmm_compress_reg_smem_bytes(int cls, int m, int rK, int c, int rb, int es) {
  return compress_layout(kRpl[cls], m, rK, c, rb, es).total;
}
// all jobs of one class; n: the largest column count rK + c or rb + min(m, rK + c)
int aifmm_compress_inline_max() { return kCompressInline; }
int aifmm_launch_compress_reg(const CompressJob* d_jobs, const CompressJob* h_jobs, int njobs, int cls, int n,
                              size_t smem, int es, cudaStream_t s) {
  if (njobs <= 0) return 0;
  if (!d_jobs && njobs > kCompressInline) return (int)cudaErrorInvalidValue;
  if (!valid_es(es) || cls < 0 || cls >= kClasses || 4 * n > qr_threads(kRpl[cls])) return (int)cudaErrorInvalidValue;
  switch (kRpl[cls]) {
#define AIFMM_CASE(R)                                                           \
    case R:                                                                     \
      return es == 16 ? launch_compress_reg<double2, R>(d_jobs, h_jobs, njobs, n, smem, s) \
                      : launch_compress_reg<float2, R>(d_jobs, h_jobs, njobs, n, smem, s);
    AIFMM_CASE(5) AIFMM_CASE(9) AIFMM_CASE(16) AIFMM_CASE(24) AIFMM_CASE(36)
#undef AIFMM_CASE
  }
  return (int)cudaErrorInvalidValue;
}
