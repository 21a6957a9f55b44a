// k_qr.cu -- batched column-pivoted QR factorisations, one CTA per block (qr.cuh).
#include <cstring>

#include "qr.cuh"

namespace {

constexpr int kQrInline = 12;
using QrInline = Inline<kQrInline * sizeof(QRJob)>;

template <typename C, int RPL>
__global__ void __launch_bounds__(qr_threads(RPL)) qr_factor_reg_kernel(const QRJob* __restrict__ jobs,
                                                                        const __grid_constant__ QrInline inl) {
  extern __shared__ double2 qsm[];
  pdl_begin();
  const QRJob J = jobs ? jobs[blockIdx.x] : reinterpret_cast<const QRJob*>(inl.b)[blockIdx.x];
  pdl_wait();
  C* a = static_cast<C*>(J.a);
  qr_reg_body<C, RPL>(J.m, J.n, [&](int row, int slot) { return a[row + (size_t)slot * J.lda]; }, a, J.lda,
                      static_cast<C*>(J.tau), J.perm, true, J.thr, J.info, J.maxpiv, reinterpret_cast<char*>(qsm));
}

template <typename C>
__global__ void __launch_bounds__(kT) qr_factor_smem_kernel(const QRJob* __restrict__ jobs) {
  extern __shared__ double2 qsm[];
  const QRJob J = jobs[blockIdx.x];
  qr_smem_body<C>(J, reinterpret_cast<C*>(qsm));
}

template <typename C, int RPL>
int launch_qr_reg(const QRJob* d_jobs, const QRJob* h_jobs, int njobs, int n, size_t smem, cudaStream_t s) {
  static SmemLimit attr;
  if (const int e = smem_limit(qr_factor_reg_kernel<C, RPL>, attr)) return e;
  QrInline inl;
  if (!d_jobs) memcpy(inl.b, h_jobs, sizeof(QRJob) * njobs);
  return launch_chain(qr_factor_reg_kernel<C, RPL>, dim3(njobs), threads_for(n), smem, s, d_jobs, inl);
}
}  // namespace

int aifmm_qr_class(int m, int n) { return qr_class(m, n); }
int aifmm_qr_inline_max() { return kQrInline; }
// all jobs of one class, at most n columns each
int aifmm_launch_qr_factor_reg(const QRJob* d_jobs, const QRJob* h_jobs, int njobs, int cls, int n, int es,
                               cudaStream_t s) {
  if (njobs <= 0) return 0;
  if (!d_jobs && njobs > kQrInline) return (int)cudaErrorInvalidValue;
  if (!valid_es(es) || cls < 0 || cls >= kClasses || 4 * n > qr_threads(kRpl[cls])) return (int)cudaErrorInvalidValue;
  const size_t smem = qr_reg_smem_bytes(kRpl[cls], n, std::min(4 * kRpl[cls], n), es) + 64;
  switch (kRpl[cls]) {
#define AIFMM_CASE(R)                                                     \
    case R:                                                               \
      return es == 16 ? launch_qr_reg<double2, R>(d_jobs, h_jobs, njobs, n, smem, s) \
                      : launch_qr_reg<float2, R>(d_jobs, h_jobs, njobs, n, smem, s);
    AIFMM_CASE(5) AIFMM_CASE(9) AIFMM_CASE(16) AIFMM_CASE(24) AIFMM_CASE(36)
#undef AIFMM_CASE
  }
  return (int)cudaErrorInvalidValue;
}
size_t aifmm_qr_smem_bytes(int m, int n, int es) {
  if (n > 1024) return ~size_t(0);  // pivot keys hold a column index below 1024
  return (size_t)es * ((size_t)qr_smem_ld(m) * n + (size_t)kW * m) +
         sizeof(double) * (3 * (size_t)n + (size_t)std::min(m, n)) + sizeof(int) * 2 * (size_t)n;
}
int aifmm_launch_qr_factor_smem(const QRJob* d_jobs, int njobs, size_t smem, int es, cudaStream_t s) {
  if (njobs <= 0) return 0;
  if (!valid_es(es)) return (int)cudaErrorInvalidValue;
  static SmemLimit attr[2];
  if (es == 16) {
    if (const int e = smem_limit(qr_factor_smem_kernel<double2>, attr[0])) return e;
    qr_factor_smem_kernel<double2><<<njobs, kT, smem, s>>>(d_jobs);
  } else {
    if (const int e = smem_limit(qr_factor_smem_kernel<float2>, attr[1])) return e;
    qr_factor_smem_kernel<float2><<<njobs, kT, smem, s>>>(d_jobs);
  }
  return (int)cudaGetLastError();
}
