// Shared definitions of the B200 propagation library: complex helpers, error plumbing
// and launch constants.  Complex numbers are double2 (x = re, y = im), the memory layout
// of NumPy's complex128, or float2 (complex64) in the mixed-precision form.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sp {

__host__ __device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__host__ __device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__host__ __device__ __forceinline__ double2 cscale(double s, double2 a) {
  return make_double2(s * a.x, s * a.y);
}
__host__ __device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
// multiply by -i (forward) or +i (inverse): exact
__host__ __device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }
__host__ __device__ __forceinline__ double2 mul_pi(double2 a) { return make_double2(-a.y, a.x); }
// complex division a / b, Smith's algorithm (one scaling, robust to overflow)
__host__ __device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
  if (fabs(b.x) >= fabs(b.y)) {
    double r = b.y / b.x, d = b.x + b.y * r;
    return make_double2((a.x + a.y * r) / d, (a.y - a.x * r) / d);
  }
  double r = b.x / b.y, d = b.x * r + b.y;
  return make_double2((a.x * r + a.y) / d, (a.y * r - a.x) / d);
}
// the same operations on complex64
__host__ __device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  return make_float2(a.x + b.x, a.y + b.y);
}
__host__ __device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return make_float2(a.x - b.x, a.y - b.y);
}
__host__ __device__ __forceinline__ float2 cscale(float s, float2 a) {
  return make_float2(s * a.x, s * a.y);
}
__host__ __device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__host__ __device__ __forceinline__ float2 mul_mi(float2 a) { return make_float2(a.y, -a.x); }
__host__ __device__ __forceinline__ float2 mul_pi(float2 a) { return make_float2(-a.y, a.x); }

// the complex type of a real type, and conversions between the two precisions
template <class R> struct complex_of;
template <> struct complex_of<double> { using type = double2; };
template <> struct complex_of<float> { using type = float2; };
template <class R> using cplx = typename complex_of<R>::type;

template <class C> __host__ __device__ __forceinline__ C to_c(double2 v);
template <> __host__ __device__ __forceinline__ double2 to_c<double2>(double2 v) { return v; }
template <> __host__ __device__ __forceinline__ float2 to_c<float2>(double2 v) {
  return make_float2((float)v.x, (float)v.y);
}
__host__ __device__ __forceinline__ double2 to_d2(double2 v) { return v; }
__host__ __device__ __forceinline__ double2 to_d2(float2 v) { return make_double2(v.x, v.y); }

// ---- a single run's chain of short kernels: each is launched as the last CTAs of the one before it
// end (programmatic dependent launch) and waits here, before its first access to global memory,
// for that one's end and its writes.  Every kernel of the chain waits, so each sees the writes of
// all before it.  A kernel launched in the ordinary way passes straight through.  It saves a
// launch's latency per kernel, about 1 us of 5.
// No kernel triggers the next one earlier (griddepcontrol.launch_dependents): CTAs that wait hold
// their place on an SM, the next kernels' are packed onto the first SMs that free up, and other
// streams find none.  With the trigger ahead of the wait, the whole chain resident at once, 24
// attempts of eight mixed modes, rows of 4 096, took 2.28 ms (2.02 in ordinary launches, 1.75
// now), and evaluations of four mixed modes, rows of 32 768, of three workspaces in turn 48.2 us
// each (46.6; 40.3).  Over 128 sizes the chain was 0.89 to 1.44 times as fast as ordinary
// launches with that trigger, and is 1.06 to 1.55 times as fast without.
// Such a kernel runs beside the one that writes its inputs, and non-coherent loads are not ordered
// after the wait: __ldg and const __restrict__ are for tables written at workspace creation alone,
// what an earlier kernel of the chain wrote is read by plain loads or __ldcg.
__device__ __forceinline__ void await_previous_kernel() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// launches a kernel that begins with await_previous_kernel, in clusters of `cluster` CTAs along x
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t shm, int cluster,
                                  cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = shm;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// exp of a complex number
__device__ __forceinline__ double2 cexp(double2 z) {
  double e = exp(z.x), s, c;
  sincos(z.y, &s, &c);
  return make_double2(e * c, e * s);
}

// Largest fine-grid length one response-column CTA holds; longer rows use a cluster.
constexpr int kColumnSpan = 4096;
constexpr int kColumnThreads = 512;
constexpr int kMaxModes = 8;   // modal route columns handled by the projection kernel
constexpr int kMaxTaps = 16;   // band-rule half-width K + 1

}  // namespace sp
