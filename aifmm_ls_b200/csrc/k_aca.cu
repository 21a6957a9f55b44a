// k_aca.cu -- batched partially pivoted ACA skeletonisation (K3).
//
// Replaces LowRank::ACA_only_nodes (ACA.hpp:368-577) as called by
// getNodes_outgoing_box / getNodes_incoming_box (FMM2DTree_find_error.hpp:1230-1336).
// One cluster of CTAs per (box, direction); all boxes of a level in one launch.
//
// The reference has two mirror-image branches: rows first when N1 < N2
// (ACA.hpp:397-481), columns first otherwise (:482-568).  Both are the same
// procedure on A or A^T, written here once in terms of a "primary" index set
// (the one scanned first) and a "secondary" one:
//   * scan primary indices in order for the first vector whose largest entry
//     over the secondary set exceeds tol_robust = 1e-12 (ACA.hpp:399-413);
//   * v = P / P[pivot], u = S (unmodified first column / row);
//   * loop while |P[s_piv]| > tol, |S[p_next]| > tol, |prev - normS| >= tol*prev,
//     rank < min(N1, N2): residual P and S against the previous terms, pivots
//     = first maximum of |.| over the remaining indices in ascending order
//     (ACA.hpp:27-40), stop when |u| or |v| < tol_robust;
//   * normS bookkeeping exactly as ACA.hpp:472-478 (the sum over l includes the
//     new term, prev_normS is not updated when the rank becomes 2).
// The unmodified rows (Ar) or columns (Ac) are the outputs the solver keeps.
#include <cfloat>
#include "aca_cluster.h"
#include "kernels.h"
#include "entry.cuh"


namespace {

// A job runs on a cluster of CTAs of 128 threads.  Thread g of the cluster owns the
// positions g, g + size * 128, ... of both index sets: it computes the entries there,
// their residuals, their magnitudes and the quotients by the pivot, all through global
// memory.  Maxima, first indices and norms are folded in each CTA and exchanged through
// the cluster's shared memory; every CTA then holds the same values, takes the same
// decisions and meets the others at the same barriers.
// What bounds it: the 61 orders of an entry, a serial chain of FP64 (34% of the FP64 rate
// at the leaves of depth 4, 17% at the level above), one primary vector after the other.
// With one CTA of 256 threads a job, and every row outside the contrast's support
// evaluated in search of a first vector, the assemblies' ACA took 2.5 ms (depth 3), 26.7
// (depth 4, 8 x 8 nodes, a disk), 37 (depth 5) and 108 ms (depth 6, a narrow Gaussian);
// now 1.07, 9.4, 28 and 17 ms.
constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCluster = kAcaMaxCluster;
constexpr int kMag = 4;      // magnitudes a thread keeps in shared memory (the rest: computed twice)
constexpr int kCoef = 32;   // coefficients of a residual held in shared memory (the rest: global memory)
typedef unsigned long long u64;

struct Shared {
  double mag[kMag][kThreads];
  double2 coef[kCoef];
  double hyp[kThreads];
  u64 key[kWarps];
  int first[kWarps];
  double sum[2][kWarps];
  // one value of each CTA of the cluster; a slot is written again only after two barriers
  u64 xkey[2][kMaxCluster], xfirst[2][kMaxCluster], xsum[2][kMaxCluster];
};

struct Cluster {
  int rank, size;
  // all CTAs of the job, and what they wrote before
  __device__ __forceinline__ void sync() const {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
  }
  // this CTA's value into slot[rank] of every CTA (threads 0 .. size - 1 of a CTA)
  __device__ __forceinline__ void put(u64* slot, u64 v) const {
    if ((int)threadIdx.x < size) {
      const unsigned a = (unsigned)__cvta_generic_to_shared(slot + rank);
      unsigned r;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(threadIdx.x));
      asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(r), "l"(v) : "memory");
    }
  }
};

// One vector of the cross: positions [0, n) of one index set against a fixed index of
// the other one.
struct Side {
  const int* var;       // the indices that vary
  int n;
  double2* terms;       // the terms' vectors along this set (rows of n)
  unsigned char* rem;   // remaining pivots
  bool vary_rows;       // var are rows of the matrix
  bool keep;            // unmodified vectors are outputs
};

struct Job {
  Side side[2];         // 0: along the secondary set (P, V), 1: along the primary set (S, U)
  double2* out;
  int want_rows, rmax;
};

// The vector with the index `fixed` against side a: the entries, less the terms before it
// (rank of them, coefficients from sh.coef and coef_at), into x.  Returns the largest
// magnitude among the thread's remaining positions (-1: none); *sum gets its |x|^2.
// Not inlined: one copy of the entry for both sides keeps the loop in the instruction cache.
template <int ENX>
__device__ __noinline__ double produce(const Job& J, int a, int fixed, int rank, const double2* coef_at, size_t coef_ld,
                                       double2* x, int drop, double floor, const EntryCtx& ctx, int g, int gn, Shared& sh,
                                       double* sum) {
  const Side& A = J.side[a];
  const int n = A.n;
  double best = -1.0, acc = 0.0;
  int k = 0;
  for (int t = g; t < n; t += gn, ++k) {
    const int v = A.var[t];
    double2 e = lsa_entry<true, ENX>(A.vary_rows ? v : fixed, A.vary_rows ? fixed : v, ctx, floor);
    if (A.keep) {
      if (J.want_rows) J.out[rank + (size_t)t * J.rmax] = e; else J.out[t + (size_t)rank * n] = e;
    }
    const double2* w = A.terms + t;
    for (int l = 0; l < rank; ++l, w += n) {
      const double2 c = l < kCoef ? sh.coef[l] : coef_at[l * coef_ld];
      e = csub(e, cmul_f<1, 2>(c, *w));
    }
    x[t] = e;
    acc += cabs2(e);
    if (t == drop) A.rem[t] = 0;
    const double m = A.rem[t] ? hypot(e.x, e.y) : -1.0;
    if (k < kMag) sh.mag[k][threadIdx.x] = m;
    if (m > best) best = m;  // no NaN
  }
  *sum = acc;
  return best;
}

// Pivot choice of ACA.hpp:27-40 with a relative tie tolerance: the first index whose
// magnitude is within kPivotTie of the maximum (the first maximum when values differ by
// more).  Magnitudes are not negative, so their bits order as integers do: 0 is "none".
constexpr double kPivotTie = 1e-11;
__device__ __forceinline__ void post_max(double best, u64* slot, const Cluster& C, Shared& sh) {
  const u64 key = best >= 0.0 ? (u64)__double_as_longlong(best) + 1 : 0;
  const unsigned hi = (unsigned)(key >> 32);
  const unsigned mhi = __reduce_max_sync(0xffffffffu, hi);
  const unsigned mlo = __reduce_max_sync(0xffffffffu, hi == mhi ? (unsigned)key : 0u);
  if ((threadIdx.x & 31) == 0) sh.key[threadIdx.x >> 5] = (u64)mhi << 32 | mlo;
  __syncthreads();
  u64 top = sh.key[0];
#pragma unroll
  for (int k = 1; k < kWarps; ++k) top = max(top, sh.key[k]);
  C.put(slot, top);
}
// after a barrier of the cluster: the first position of x within the tie of the maximum
__device__ __forceinline__ void post_first(const u64* maxima, const double2* x, const Side& A, u64* slot, int g, int gn,
                                           const Cluster& C, Shared& sh) {
  u64 top = 0;
  for (int k = 0; k < C.size; ++k) top = max(top, maxima[k]);
  unsigned first = 0x7fffffffu;
  if (top) {
    const double cut = __longlong_as_double((long long)(top - 1)) * (1.0 - kPivotTie);
    int k = 0;
    for (int t = g; t < A.n; t += gn, ++k) {
      double v;
      if (k < kMag) v = sh.mag[k][threadIdx.x];
      else v = A.rem[t] ? hypot(x[t].x, x[t].y) : -1.0;
      if (v >= 0.0 && v >= cut) { first = t; break; }
    }
  }
  first = __reduce_min_sync(0xffffffffu, first);
  if ((threadIdx.x & 31) == 0) sh.first[threadIdx.x >> 5] = (int)first;
  __syncthreads();
  int f = sh.first[0];
#pragma unroll
  for (int k = 1; k < kWarps; ++k) f = min(f, sh.first[k]);
  C.put(slot, (u64)f);
}
// after another one; -1 if no position remains
__device__ __forceinline__ int first_of(const u64* firsts, const Cluster& C) {
  int f = (int)firsts[0];
  for (int k = 1; k < C.size; ++k) f = min(f, (int)firsts[k]);
  return f == 0x7fffffff ? -1 : f;
}
__device__ __forceinline__ void post_sums(double a, double b, const Cluster& C, Shared& sh) {
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
  }
  if ((threadIdx.x & 31) == 0) { sh.sum[0][threadIdx.x >> 5] = a; sh.sum[1][threadIdx.x >> 5] = b; }
  __syncthreads();
  a = b = 0.0;
#pragma unroll
  for (int k = 0; k < kWarps; ++k) { a += sh.sum[0][k]; b += sh.sum[1][k]; }
  C.put(sh.xsum[0], (u64)__double_as_longlong(a));
  C.put(sh.xsum[1], (u64)__double_as_longlong(b));
}
__device__ __forceinline__ double sum_of(const u64* sums, const Cluster& C) {
  double r = 0.0;
  for (int k = 0; k < C.size; ++k) r += __longlong_as_double((long long)sums[k]);
  return r;
}

// Dots of the rows [0, rank) of X (n entries each) with row rank - 1: two rows a warp,
// the warps of the whole cluster
__device__ void row_dots(const double2* X, int n, int rank, double2* out, int gw, int nw) {
  const int lane = threadIdx.x & 31;
  const double2* xn = X + (size_t)(rank - 1) * n;
  for (int l = 2 * gw; l < rank; l += 2 * nw) {
    const int l1 = l + 1 < rank ? l + 1 : l;
    const double2* x0 = X + (size_t)l * n;
    const double2* x1 = X + (size_t)l1 * n;
    double2 d0 = make_double2(0.0, 0.0), d1 = d0;
    for (int t = lane; t < n; t += 32) {
      const double2 y = xn[t];
      d0 = cfmac(x0[t], y, d0);
      d1 = cfmac(x1[t], y, d1);
    }
    for (int o = 16; o > 0; o >>= 1) {
      d0.x += __shfl_down_sync(0xffffffffu, d0.x, o); d0.y += __shfl_down_sync(0xffffffffu, d0.y, o);
      d1.x += __shfl_down_sync(0xffffffffu, d1.x, o); d1.y += __shfl_down_sync(0xffffffffu, d1.y, o);
    }
    if (lane == 0) { out[l] = d0; out[l1] = d1; }
  }
}

__global__ void __launch_bounds__(kThreads, 4) aca_kernel(const AcaJob* __restrict__ jobs, double tol,
                                                          const __grid_constant__ EntryCtx ctx, int csize) {
  const AcaJob& A = jobs[blockIdx.x / csize];
  const Cluster C{(int)(blockIdx.x % csize), csize};
  __shared__ Shared sh;
  __shared__ Job J;
  const double tol_robust = 1e-12;  // ACA.hpp:23
  const int tid = threadIdx.x;
  const int g = C.rank * kThreads + tid, gn = csize * kThreads;  // in the cluster
  const int gw = g >> 5, nw = gn >> 5;
  const bool lead = g == 0;
  const bool rows_first = A.n1 < A.n2;
  const int np = rows_first ? A.n1 : A.n2;   // primary count
  const int ns = rows_first ? A.n2 : A.n1;   // secondary count
  const int rmax = min(A.n1, A.n2);
  const int* prim = rows_first ? A.rows : A.cols;
  const int* sec = rows_first ? A.cols : A.rows;
  double2 *const P = A.P, *const U = A.U, *const V = A.V, *const dots_u = A.dots_u, *const dots_v = A.dots_v;
  int *const prim_bases = A.prim_bases, *const sec_bases = A.sec_bases, *const rank_out = A.rank;
  if (tid == 0) {
    // the outputs' side: in rows-first mode rows are primary vectors
    const bool keepP = (A.want_rows != 0) == rows_first;
    J.side[0] = Side{sec, ns, V, A.remS, !rows_first, keepP};
    J.side[1] = Side{prim, np, U, A.remP, rows_first, !keepP};
    J.out = A.out; J.want_rows = A.want_rows; J.rmax = rmax;
  }
  if (lead) { rank_out[0] = 0; rank_out[1] = rows_first ? 1 : 2; }
  if (rmax == 0) return;
  for (int t = g; t < np; t += gn) A.remP[t] = 1;
  for (int t = g; t < ns; t += gn) A.remS[t] = 1;
  C.sync();
  // ---- first primary vector with a non-negligible entry: entries that are bounded by
  // tol_robust need not be known for that
  double norm = 0.0;
  int p0 = -1, spiv = -1;
  for (int l = 0; l < np; ++l) {
    const double best = produce<2>(J, 0, prim[l], 0, nullptr, 0, P, -1, tol_robust, ctx, g, gn, sh, &norm);
    post_max(best, sh.xkey[0], C, sh);
    C.sync();
    u64 top = 0;
    for (int k = 0; k < csize; ++k) top = max(top, sh.xkey[0][k]);
    const bool found = top && __longlong_as_double((long long)(top - 1)) > tol_robust;
    post_first(sh.xkey[0], P, J.side[0], sh.xfirst[0], g, gn, C, sh);
    C.sync();
    if (found) { p0 = l; spiv = first_of(sh.xfirst[0], C); break; }
  }
  if (p0 < 0) return;  // rank 0
  if (!rows_first) {  // a column: its entries below tol_robust too
    produce<2>(J, 0, prim[p0], 0, nullptr, 0, P, -1, kEntryFloor, ctx, g, gn, sh, &norm);
    C.sync();
  }
  // v = P / P[spiv]; U[0] = S = secondary vector at spiv
  const double2 piv0 = P[spiv];
  double pivP = hypot(piv0.x, piv0.y);
  for (int s = g; s < ns; s += gn) {
    V[s] = cdiv(P[s], piv0);
    if (s == spiv) J.side[0].rem[s] = 0;
  }
  double best = produce<2>(J, 1, sec[spiv], 0, nullptr, 0, U, p0, kEntryFloor, ctx, g, gn, sh, &norm);
  if (lead) { prim_bases[0] = p0; sec_bases[0] = spiv; }
  post_max(best, sh.xkey[1], C, sh);
  C.sync();
  post_first(sh.xkey[1], U, J.side[1], sh.xfirst[1], g, gn, C, sh);
  C.sync();
  int rank = 1;
  double normS = 0.0, prev = DBL_MAX;
  while (true) {
    // next primary pivot: max |S| over remaining primary indices
    const int pnext = max(first_of(sh.xfirst[1], C), 0);
    const double2 last = U[(size_t)(rank - 1) * np + pnext];
    const double sp = hypot(last.x, last.y);
    if (!(pivP > tol && sp > tol && fabs(prev - normS) >= tol * prev && rank < rmax)) break;
    // ---- primary vector at pnext, residual against previous terms
    for (int l = tid; l < min(rank, kCoef); l += kThreads) sh.coef[l] = U[(size_t)l * np + pnext];
    __syncthreads();
    best = produce<1>(J, 0, prim[pnext], rank, U + pnext, np, P, -1, kEntryFloor, ctx, g, gn, sh, &norm);
    post_max(best, sh.xkey[0], C, sh);
    C.sync();
    post_first(sh.xkey[0], P, J.side[0], sh.xfirst[0], g, gn, C, sh);
    C.sync();
    const int snew = max(first_of(sh.xfirst[0], C), 0);
    const double2 pivot = P[snew];
    for (int l = tid; l < min(rank, kCoef); l += kThreads) sh.coef[l] = V[(size_t)l * ns + snew];
    double vn2 = 0.0, un2;
    for (int s = g; s < ns; s += gn) {
      const double2 v = cdiv(P[s], pivot);
      V[(size_t)rank * ns + s] = v;
      vn2 += cabs2(v);
      if (s == snew) J.side[0].rem[s] = 0;
    }
    __syncthreads();
    best = produce<1>(J, 1, sec[snew], rank, V + snew, ns, U + (size_t)rank * np, pnext, kEntryFloor, ctx, g, gn, sh, &un2);
    post_max(best, sh.xkey[1], C, sh);
    post_sums(un2, vn2, C, sh);
    C.sync();
    const double un = sqrt(sum_of(sh.xsum[0], C)), vn = sqrt(sum_of(sh.xsum[1], C));
    if (un < tol_robust || vn < tol_robust) break;  // term rejected, bases not committed
    if (lead) { prim_bases[rank] = pnext; sec_bases[rank] = snew; }
    pivP = hypot(pivot.x, pivot.y);
    post_first(sh.xkey[1], U + (size_t)rank * np, J.side[1], sh.xfirst[1], g, gn, C, sh);
    ++rank;
    // normS update (ACA.hpp:472-478): dots of every stored term with the new one
    row_dots(V, ns, rank, dots_v, gw, nw);
    row_dots(U, np, rank, dots_u, nw - 1 - gw, nw);
    C.sync();
    if (rank != 2) prev = normS;
    double ns_ = normS * normS + (un * vn) * (un * vn);
    for (int l0 = 0; l0 < rank; l0 += kThreads) {  // a lane each, summed in their order
      if (l0) __syncthreads();
      if (l0 + tid < rank) {
        const double2 pr = cmul(dots_u[l0 + tid], dots_v[l0 + tid]);
        sh.hyp[tid] = hypot(pr.x, pr.y);
      }
      __syncthreads();
      for (int l = 0; l < min(rank - l0, kThreads); ++l) ns_ += 2 * sh.hyp[l];
    }
    normS = sqrt(ns_);
  }
  if (lead) rank_out[0] = rank;
}

}  // namespace

int aifmm_launch_aca(const AcaJob* d_jobs, int njobs, long level_jobs, double tol, const EntryCtx& ctx,
                     cudaStream_t stream) {
  if (njobs <= 0) return 0;
  const int csize = aca_cluster_size(level_jobs);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(njobs * csize));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)csize;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, aca_kernel, d_jobs, tol, ctx, csize);
}
