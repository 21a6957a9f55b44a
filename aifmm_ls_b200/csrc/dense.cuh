// dense.cuh -- helpers shared by the dense kernels (k_dense.cu, k_qr.cu).
#pragma once
#include <cfloat>
#include "kernels.h"
#include "smem_limit.h"

namespace {

constexpr int kT = 256;
constexpr int kW = kT / 32;
constexpr double kPivotTie = 1e-11;  // same pivot tie tolerance as the ACA

// Real-type constants of the two forms: machine epsilon, the smallest normal
// number, and the range inside which a product may be inverted directly.
template <typename R> struct rl;
template <> struct rl<double> {
  static constexpr double eps = DBL_EPSILON, tiny = DBL_MIN, lo = 1e-290, hi = 1e290;
};
template <> struct rl<float> {
  static constexpr float eps = FLT_EPSILON, tiny = FLT_MIN, lo = 1e-35f, hi = 1e35f;
};

// Norms, reflector scalars and pivot reciprocals are computed in double for both
// forms: complex64 blocks of the contrast's far corners hold values near 1e-25,
// whose squares underflow FP32 and whose reciprocals overflow it.  The O(m n)
// column updates stay in the blocks' own precision.
__device__ __forceinline__ double cabs2d(double2 a) { return cabs2(a); }
__device__ __forceinline__ double cabs2d(float2 a) { const double x = a.x, y = a.y; return x * x + y * y; }
__device__ __forceinline__ double2 c2d(double2 a) { return a; }
__device__ __forceinline__ double2 c2d(float2 a) { return make_double2(a.x, a.y); }

// Products with their rounding written out.  Which of a complex product's two real
// products an FMA absorbs is otherwise the compiler's choice, and differs from one
// kernel to the next; a block's factors must not depend on the kernel that takes it.
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// a b: the first products are fused
template <typename C>
__device__ __forceinline__ C cmul_p(C a, C b) {
  C r;
  r.x = rfma(a.x, b.x, -rmul(a.y, b.y));
  r.y = rfma(a.x, b.y, rmul(a.y, b.x));
  return r;
}
// a b for the reflector's coefficient a: the second product of the imaginary part is fused
template <typename C>
__device__ __forceinline__ C cmul_t(C a, C b) {
  C r;
  r.x = rfma(a.x, b.x, -rmul(a.y, b.y));
  r.y = rfma(a.y, b.x, rmul(a.x, b.y));
  return r;
}
__device__ __forceinline__ double cabs2_p(double2 a) { return __fma_rn(a.x, a.x, __dmul_rn(a.y, a.y)); }
__device__ __forceinline__ double cabs2_p(float2 a) { return cabs2_p(make_double2(a.x, a.y)); }

// Programmatic dependent launch.  The kernels of an elimination step or a solve wave
// are a chain of launches of a few microseconds each; a kernel launched this way is
// set up (and reads its descriptors) while the one before it still runs, and waits in
// pdl_wait until that one has finished and its writes are visible.  Every kernel
// launched with launch_chain calls both, pdl_wait before its first access to memory that
// another kernel writes: then a kernel that has finished implies that all before it
// have.
__device__ __forceinline__ void pdl_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... P, typename... A>
int launch_chain(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Descriptors of a small batch travel in the kernel's parameters: no copy between the
// launches of a chain.
template <int BYTES>
struct Inline {
  alignas(16) unsigned char b[BYTES];
};

// the element size of a batch: 16 (complex128) or 8 (complex64)
inline bool valid_es(int es) { return es == 16 || es == 8; }

}  // namespace
