// k_entries.cu -- batched matrix-entry assembly (K1).
//
// Replaces kernel::getRow / getCol / getMatrix (kernel.hpp:54-86) and the block
// assemblies built on them: leaf P2P blocks (FMM2DTree_find_error.hpp:1729-1741),
// M2L blocks (:1338-1361), the skeleton blocks of get_L2P_P2M_box (:1105-1128),
// and the dense product of the find_error fixture generator
// (FMM2DTree_gen_rhs_x.hpp:2864-2871).
#include <algorithm>

#include "kernels.h"
#include "entry.cuh"


namespace {

__global__ void block_entries_kernel(const BlockDesc* __restrict__ d, const long long* __restrict__ off, int nd,
                                     long long total, EntryCtx ctx) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    int lo = 0, hi = nd - 1;
    while (lo < hi) {  // last descriptor with off <= e
      int mid = (lo + hi + 1) >> 1;
      if (off[mid] <= e) lo = mid; else hi = mid - 1;
    }
    const BlockDesc b = d[lo];
    const long long loc = e - off[lo];
    const int r = (int)(loc % b.nr), c = (int)(loc / b.nr);
    double2 v = lsa_entry(__ldg(&b.rows[r]), __ldg(&b.cols[c]), ctx);
    if (b.adjoint) b.out[c + (size_t)r * b.ldo] = cconj(v);
    else b.out[r + (size_t)c * b.ldo] = v;
  }
}

__global__ void list_entries_kernel(const int* __restrict__ I, const int* __restrict__ J, long n, double2* out,
                                    EntryCtx ctx) {
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x)
    out[t] = lsa_entry(I[t], J[t], ctx);
}

// ---- y(:, s) = A x(:, s) for nrhs <= 8 columns (x, y: N x nrhs column-major)
//
// A far entry is a 121-term series in the source point's coefficients M(:, j)
// whose Hankel values and angles depend on the target point and the source LEAF
// only.  So the sources of a leaf are summed first: m(n, s) = sum_j M(n, j) x(j, s)
// (moments_kernel), and one series per (target, leaf) replaces one per entry --
// rank times fewer Bessel recurrences.  Rows whose far entries are all zero by the
// entries' own bound have no series; in the others the far entries below 1e-16, zero
// in the matrix, are part of the sum.
//   sum_n H_n(R) e^{in th} m_n = sum_{n >= 0} (J_n + i Y_n) (p_n cos n th + q_n sin n th)
//   p_n = m_n + (-1)^n m_{-n},  q_n = i (m_n - (-1)^n m_{-n}),  p_0 = m_0,  q_0 = 0
// What bounds it: latency and issue of the FP64 recurrences (about 1,900 double
// instructions per target, leaf and one right-hand side; the moments are warp-
// uniform reads of shared memory; FP64 pipe 47% busy).  36,864 unknowns, one right-hand side, through
// dense_matvec with host buffers: 958 ms with a series per entry, 3.2 ms with a
// series per leaf; 2,304 unknowns: 4.4 ms and 0.13 ms; 256 unknowns: 99 us and 63 us.
//
// The recurrences run unnormalised, between 1e-250 and 1e212, and a moment multiplies them:
// so a leaf's sources are divided by the power of two of their largest part, which comes
// back exactly where the normalised sums are added up (a vector of 1e100 or 1e-100 would
// overflow or vanish on the way).
constexpr int kMvRows = 128;
constexpr int kMvMaxRhs = 8;
constexpr size_t kMvMomentBytes = size_t(64) << 20;  // moments of one chunk of leaves
struct Moment { double2 p, q; };
// of a leaf and a right-hand side: the orders 0 .. 60, then the power of two (in p.x)
constexpr int kMoments = AIFMM_SERIES + 2;

__global__ void __launch_bounds__(128) moments_kernel(const double2* __restrict__ x, Moment* __restrict__ mom, int N,
                                                      int nrhs, int leaf0, int rank, const double2* __restrict__ M) {
  const int leaf = leaf0 + blockIdx.x;
  __shared__ int s_exp[kMvMaxRhs];
  // the exponents of the leaf's largest parts, a warp a right-hand side
  for (int s = threadIdx.x >> 5; s < nrhs; s += blockDim.x >> 5) {
    unsigned top = 0;
    for (int j = threadIdx.x & 31; j < rank; j += 32) {
      const double2 xv = __ldg(&x[(size_t)leaf * rank + (size_t)s * N + j]);
      top = max(top, max((unsigned)__double2hiint(xv.x) & 0x7fffffffu, (unsigned)__double2hiint(xv.y) & 0x7fffffffu));
    }
    top = __reduce_max_sync(0xffffffffu, top) >> 20;
    // infinities and NaN as they are; 2^-1000 .. 2^1000: its inverse is a double too
    if ((threadIdx.x & 31) == 0) s_exp[s] = top == 0x7ff ? 0 : max(-1000, min(1000, (int)top - 1023));
  }
  __syncthreads();
  for (int t = threadIdx.x; t < kMoments * nrhs; t += blockDim.x) {
    const int n = t / nrhs, s = t - n * nrhs;
    Moment* const out = mom + ((size_t)blockIdx.x * kMoments + n) * nrhs + s;
    if (n > AIFMM_SERIES) {
      const double2 two = make_double2(__hiloint2double((1023 + s_exp[s]) << 20, 0), 0.0);
      *out = Moment{two, make_double2(0.0, 0.0)};
      continue;
    }
    const double2* xs = x + (size_t)leaf * rank + (size_t)s * N;
    const double down = __hiloint2double((1023 - s_exp[s]) << 20, 0);
    double2 a = make_double2(0.0, 0.0), b = a;
    for (int j = 0; j < rank; ++j) {
      const double2* Mc = M + (size_t)j * (2 * AIFMM_SERIES + 1) + AIFMM_SERIES;
      const double2 xv = cscale(__ldg(&xs[j]), down);
      a = cfma(__ldg(&Mc[n]), xv, a);
      b = cfma(__ldg(&Mc[-n]), xv, b);
    }
    Moment o;
    if (n == 0) {
      o.p = a;
      o.q = make_double2(0.0, 0.0);
    } else {
      if (n & 1) b = cneg(b);
      const double2 d = csub(a, b);
      o.p = cadd(a, b);
      o.q = make_double2(-d.y, d.x);
    }
    *out = o;
  }
}

// Coefficients of the Neumann sums that give Y_0 and Y_1 from the J values of
// Miller's recurrence: even m contribute (-1)^(m/2) / (m/2) J_m to the first, odd
// m contribute (-1)^((m+1)/2) (2/(m+1) + 2/(m-1)) J_m to the second (entry.cuh).
constexpr int kNeumann = 512;
struct NeumannTable {
  double c[kNeumann];
  constexpr NeumannTable() : c() {
    for (int m = 1; m < kNeumann; ++m) c[m] = coef(m);
  }
  __host__ __device__ static constexpr double coef(int m) {
    if (m % 2 == 0) return (m / 2 % 2 ? -1.0 : 1.0) / (m / 2);
    const int a = (m + 1) / 2;
    return (a % 2 ? -1.0 : 1.0) * (1.0 / a + (m > 1 ? 1.0 / (a - 1) : 0.0));
  }
};
__constant__ NeumannTable c_neumann = NeumannTable();

// acc[s] += sum_n H_n(R) (p_n cos n th + q_n sin n th), (dx, dy) = target - leaf centre.
// All lanes of `mask` call it together: the downward recurrence starts at the
// largest order any of them needs, so that the loop and its tables are uniform.
template <int NR>
__device__ __forceinline__ void moment_series(double dx, double dy, double kappa, const Moment* mom,
                                              unsigned mask, double2 (&acc)[NR]) {
  const double rho = sqrt(dx * dx + dy * dy);
  const double R = kappa * rho;
  const double2 e1 = make_double2(dx / rho, dy / rho);
  // e^{i 16 th}, e^{i 32 th}, e^{i 48 th} restart the rotation every 16 orders
  double2 t2 = cmul(e1, e1), t4 = cmul(t2, t2), t8 = cmul(t4, t4);
  const double2 e16 = cmul(t8, t8), e32 = cmul(e16, e16), e48 = cmul(e32, e16);
  const double big = fmax((double)AIFMM_SERIES, R);
  int N = (int)(big + 24.0 + 10.0 * cbrt(big));
  N += (N & 1);
  N = __reduce_max_sync(mask, N);
  const double inv2 = 2.0 / R;
  double jp1 = 0.0, jcur = 1.0e-250, norm = 0.0;
  double S0 = 0.0, S1 = 0.0;
  double2 a[NR];
#pragma unroll
  for (int s = 0; s < NR; ++s) a[s] = make_double2(0.0, 0.0);
  double2 e = cmul(e48, cmul(t8, t4));  // e^{i 60 th}
  // ---- downward: J_m, m = N - 1 .. 0, unnormalised
  double dk = N;  // m + 1 as a double: conversions run at a fraction of the FP64 rate
  for (int m = N - 1; m >= 0; --m, dk -= 1.0) {
    const double jnew = fma(dk * inv2, jcur, -jp1);
    jp1 = jcur;
    jcur = jnew;
    const double c = m < kNeumann ? c_neumann.c[m] : NeumannTable::coef(m);
    if (m & 1) {
      S1 = fma(c, jnew, S1);
    } else {
      norm += jnew;  // doubled at the end, where J_0 counts once
      S0 = fma(c, jnew, S0);
    }
    if (m <= AIFMM_SERIES) {
      if (m < AIFMM_SERIES) e = (m & 15) == 15 ? (m == 47 ? cmul(e48, cconj(e1)) : m == 31 ? cmul(e32, cconj(e1)) : cmul(e16, cconj(e1)))
                                               : cmul(e, cconj(e1));
#pragma unroll
      for (int s = 0; s < NR; ++s) {
        const Moment& w = mom[m * NR + s];
        const double2 p = w.p, q = w.q;
        const double jc = jnew * e.x, js = jnew * e.y;
        a[s].x = fma(p.x, jc, a[s].x); a[s].x = fma(q.x, js, a[s].x);
        a[s].y = fma(p.y, jc, a[s].y); a[s].y = fma(q.y, js, a[s].y);
      }
    }
    if ((__double2hiint(jcur) & 0x7fffffff) > 0x69800000) {  // |J| above about 1e200: rescale
      const double f = 1.0e-200;
      jcur *= f; jp1 *= f; norm *= f; S0 *= f; S1 *= f;
#pragma unroll
      for (int s = 0; s < NR; ++s) a[s] = cscale(a[s], f);
    }
  }
  const double inorm = 1.0 / (2.0 * norm - jcur);
  const double J0 = jcur * inorm, J1 = jp1 * inorm;
  S0 *= inorm; S1 *= inorm;
  // the power of two of inorm first, so that the one of the leaf meets a normalised sum
  const int hi = __double2hiint(inorm);
  const double ipow = __hiloint2double(hi & 0x7ff00000, 0);
  const double iman = __hiloint2double((hi & 0x800fffff) | 0x3ff00000, __double2loint(inorm));
#pragma unroll
  for (int s = 0; s < NR; ++s) {
    const double w = iman * mom[(AIFMM_SERIES + 1) * NR + s].p.x;
    acc[s].x = fma(a[s].x * ipow, w, acc[s].x);
    acc[s].y = fma(a[s].y * ipow, w, acc[s].y);
    a[s] = make_double2(0.0, 0.0);
  }
  // ---- upward: Y_n, n = 0 .. 60
  const double kTwoOverPi = 0.63661977236758134307553505349;
  const double kEuler = 0.57721566490153286060651209008;
  const double lg = log(0.5 * R) + kEuler;
  double yc = kTwoOverPi * (lg * J0 - 2.0 * S0);
  double yn = -kTwoOverPi / R * J0 + kTwoOverPi * (lg * J1 + S1);
  e = make_double2(1.0, 0.0);
  dk = 1.0;
  for (int n = 0; n <= AIFMM_SERIES; ++n, dk += 1.0) {
    const double jc = yc * e.x, js = yc * e.y;
#pragma unroll
    for (int s = 0; s < NR; ++s) {
      const Moment& w = mom[n * NR + s];
      const double2 p = w.p, q = w.q;
      a[s].x = fma(p.x, jc, a[s].x); a[s].x = fma(q.x, js, a[s].x);
      a[s].y = fma(p.y, jc, a[s].y); a[s].y = fma(q.y, js, a[s].y);
    }
    const double y2 = fma(dk * inv2, yn, -yc);
    yc = yn;
    yn = y2;
    e = (n & 15) == 15 ? (n == 15 ? e16 : n == 31 ? e32 : e48) : cmul(e, e1);
  }
#pragma unroll
  for (int s = 0; s < NR; ++s) {  // + i SY
    const double w = mom[(AIFMM_SERIES + 1) * NR + s].p.x;
    acc[s].x = fma(-w, a[s].y, acc[s].x);
    acc[s].y = fma(w, a[s].x, acc[s].y);
  }
}

// Each thread owns one target row and a slice of the chunk's source leaves; the
// slices are combined with atomics.  NR = nrhs, so that the accumulators stay in
// registers.
template <bool PHI, int NR>
__global__ void __launch_bounds__(kMvRows) leaf_matvec_kernel(const double2* __restrict__ x, double2* y, int N,
                                                               int leaf0, int nleaf, int leaves_per_slice,
                                                               const Moment* __restrict__ mom, EntryCtx ctx) {
  __shared__ Moment sm[kMoments * NR];
  const bool live = blockIdx.x * kMvRows + threadIdx.x < N;
  const int i = min((int)(blockIdx.x * kMvRows + threadIdx.x), N - 1);
  const int l0 = blockIdx.y * leaves_per_slice;
  const int l1 = min(nleaf, l0 + leaves_per_slice);
  const int rank = ctx.rank, li = i / rank;
  const int2 me = __ldg(&ctx.leafxy[li]);
  const double2 ri = __ldg(&ctx.pts[i]);
  const double qi = __ldg(&ctx.q[i]);
  const double kq = ctx.kappa * ctx.kappa * qi;
  // the rows whose far entries are zero in the matrix too (entry.cuh)
  const bool no_far = PHI && far_is_zero(qi, ctx, kEntryFloor);
  double2 far[NR], near[NR];
#pragma unroll
  for (int s = 0; s < NR; ++s) far[s] = near[s] = make_double2(0.0, 0.0);
  for (int l = l0; l < l1; ++l) {
    // the leaf's moments, read by every thread order by order: one load latency
    // for all of them instead of one per order
    const double2* src = reinterpret_cast<const double2*>(mom + (size_t)l * kMoments * NR);
    for (int t = threadIdx.x; t < 2 * kMoments * NR; t += kMvRows)
      reinterpret_cast<double2*>(sm)[t] = __ldg(&src[t]);
    __syncthreads();
    const int lj = leaf0 + l;
    const int2 b = __ldg(&ctx.leafxy[lj]);
    const int dx = b.x - me.x, dy = b.y - me.y;
    const bool close = dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1;
    const bool series = !close && !no_far;
    const unsigned mask = __ballot_sync(0xffffffffu, series);
    if (series) {
      const double2 c = __ldg(&ctx.leafc[lj]);
      moment_series<NR>(ri.x - c.x, ri.y - c.y, ctx.kappa, sm, mask, far);
    } else if (close) {
      for (int j = 0; j < rank; ++j) {
        const double2 a = lsa_entry<PHI>(i, lj * rank + j, ctx);
        if (a.x == 0.0 && a.y == 0.0) continue;
#pragma unroll
        for (int s = 0; s < NR; ++s) near[s] = cfma(a, __ldg(&x[(size_t)lj * rank + j + (size_t)s * N]), near[s]);
      }
    }
    __syncthreads();
  }
  if (!live) return;
#pragma unroll
  for (int s = 0; s < NR; ++s) {
    double2 v = make_double2(-0.25 * far[s].y, 0.25 * far[s].x);  // times i/4
    if (PHI) v = cscale(v, kq);
    v = cadd(v, near[s]);
    atomicAdd(&y[i + (size_t)s * N].x, v.x);
    atomicAdd(&y[i + (size_t)s * N].y, v.y);
  }
}

}  // namespace

int aifmm_launch_block_entries(const BlockDesc* d_desc, const long long* d_off, int nd, long long total,
                               const EntryCtx& ctx, cudaStream_t stream) {
  if (nd <= 0 || total <= 0) return 0;
  long long blocks = (total + 255) / 256;
  if (blocks > 148LL * 64) blocks = 148LL * 64;
  block_entries_kernel<<<(int)blocks, 256, 0, stream>>>(d_desc, d_off, nd, total, ctx);
  return (int)cudaGetLastError();
}

int aifmm_launch_list_entries(const int* I, const int* J, long n, double2* out, const EntryCtx& ctx,
                              cudaStream_t stream) {
  if (n <= 0) return 0;
  long blocks = (n + 255) / 256;
  if (blocks > 148L * 64) blocks = 148L * 64;
  list_entries_kernel<<<(int)blocks, 256, 0, stream>>>(I, J, n, out, ctx);
  return (int)cudaGetLastError();
}

// bytes of moment scratch a dense product needs: one chunk of leaves
size_t aifmm_matvec_scratch_bytes(int N, int rank, int nrhs) {
  const size_t per_leaf = sizeof(Moment) * kMoments * (size_t)nrhs;
  const size_t nleaf = (size_t)N / rank;
  return per_leaf * std::min(nleaf, std::max<size_t>(1, kMvMomentBytes / per_leaf));
}

namespace {
template <bool PHI, int NR>
void launch_leaf_matvec(dim3 grid, const double2* x, double2* y, int N, int leaf0, int nl, int lps, const Moment* mom,
                        const EntryCtx& ctx, cudaStream_t stream) {
  leaf_matvec_kernel<PHI, NR><<<grid, kMvRows, 0, stream>>>(x, y, N, leaf0, nl, lps, mom, ctx);
}
template <bool PHI>
int launch_matvec(const double2* x, double2* y, int N, int nrhs, void* scratch, const EntryCtx& ctx,
                  cudaStream_t stream) {
  if (nrhs < 1 || nrhs > kMvMaxRhs) return (int)cudaErrorInvalidValue;
  Moment* mom = static_cast<Moment*>(scratch);
  const int nleaf = N / ctx.rank;
  const int chunk = (int)(aifmm_matvec_scratch_bytes(N, ctx.rank, nrhs) / (sizeof(Moment) * kMoments * nrhs));
  const int row_blocks = (N + kMvRows - 1) / kMvRows;
  for (int leaf0 = 0; leaf0 < nleaf; leaf0 += chunk) {
    const int nl = std::min(chunk, nleaf - leaf0);
    moments_kernel<<<nl, 128, 0, stream>>>(x, mom, N, nrhs, leaf0, ctx.rank, ctx.M);
    // Rows far outside the contrast finish at once, so the slices are many more than
    // fill the chip: up to 64 CTAs for every SM, but at least 4 leaves a slice once
    // there are 8 CTAs for every SM.
    const int few = (148 * 8 + row_blocks - 1) / row_blocks, many = (148 * 64 + row_blocks - 1) / row_blocks;
    const int slices0 = std::max(1, std::min(nl, std::max(few, std::min(many, nl / 4))));
    const int lps = (nl + slices0 - 1) / slices0;
    const dim3 grid(row_blocks, (nl + lps - 1) / lps);
    switch (nrhs) {
#define AIFMM_MV_CASE(R) \
      case R: launch_leaf_matvec<PHI, R>(grid, x, y, N, leaf0, nl, lps, mom, ctx, stream); break;
      AIFMM_MV_CASE(1) AIFMM_MV_CASE(2) AIFMM_MV_CASE(3) AIFMM_MV_CASE(4)
      AIFMM_MV_CASE(5) AIFMM_MV_CASE(6) AIFMM_MV_CASE(7) AIFMM_MV_CASE(8)
#undef AIFMM_MV_CASE
    }
    const int e = (int)cudaGetLastError();
    if (e) return e;
  }
  return 0;
}
}  // namespace

int aifmm_launch_dense_matvec(const double2* x, double2* y, int N, int nrhs, void* scratch, const EntryCtx& ctx,
                              cudaStream_t stream) {
  if (nrhs > kMvMaxRhs) return (int)cudaErrorInvalidValue;
  cudaMemsetAsync(y, 0, sizeof(double2) * (size_t)N * nrhs, stream);
  return launch_matvec<true>(x, y, N, nrhs, scratch, ctx, stream);
}
int aifmm_launch_green_matvec_add(const double2* x, double2* y, int N, int nrhs, void* scratch, const EntryCtx& ctx,
                                  cudaStream_t stream) {
  return launch_matvec<false>(x, y, N, nrhs, scratch, ctx, stream);
}
