// gd_common.cuh -- shared definitions of the GB300 spectral dycore kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <cstdio>
#include <stdexcept>
#include <string>

namespace gd {

// Fortran literals without a kind suffix are single precision in the
// reference (no -fdefault-real-8, src/Makefile.conf.gfortran), so its
// constants carry float-rounded values in every build.
#define GD_FLIT(x) ((double)(float)(x))

// src/physcons.f90:17-56
struct Phys {
  static constexpr double rerth = GD_FLIT(6.3712e+6f);
  static constexpr double grav = GD_FLIT(9.80665e+0f);
  static constexpr double omega = GD_FLIT(7.2921e-5f);
  static constexpr double rd = GD_FLIT(2.8705e+2f);
  static constexpr double rv = GD_FLIT(4.6150e+2f);
  static constexpr double cp = GD_FLIT(1.0046e+3f);
  static constexpr double cvap = GD_FLIT(1.8460e+3f);
};

struct CudaError : std::runtime_error {
  explicit CudaError(const std::string& s) : std::runtime_error(s) {}
};

#define GD_CUDA(call)                                                                         \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess) {                                                                  \
      cudaGetLastError(); /* reported here: no later launch check is to see it again */       \
      throw ::gd::CudaError(std::string(#call) + ": " + cudaGetErrorString(e_) + " @" +      \
                            __FILE__ + ":" + std::to_string(__LINE__));                      \
    }                                                                                         \
  } while (0)

#define GD_LAUNCH_CHECK() GD_CUDA(cudaGetLastError())

// 2-component vector of the real type (one complex number).
template <typename R>
struct C2;
template <>
struct C2<double> {
  typedef double2 T;
};
template <>
struct C2<float> {
  typedef float2 T;
};

// two complex values in one aligned load (16 bytes FP32, 32 bytes FP64)
struct __align__(32) GdDouble4 {
  double x, y, z, w;
};
template <typename R>
struct C4;
template <>
struct C4<double> {
  typedef GdDouble4 T;
};
template <>
struct C4<float> {
  typedef float4 T;
};

template <typename R>
__host__ __device__ inline typename C2<R>::T mk2(R x, R y) {
  typename C2<R>::T v;
  v.x = x;
  v.y = y;
  return v;
}

inline int ceil_div(long a, long b) { return (int)((a + b - 1) / b); }

// Reciprocal in FP64 for kernels that the FP64 pipe (two lanes per clock and
// SM) bounds: one step of Halley's third-order iteration r (1 + e + e^2), e = 1
// - x r, on the hardware's approximation (relative error at most 1.05 2^-20,
// measured over every mantissa it tells apart; e^3 is below 2^-59): three
// multiply-adds, within 1.004 roundings (2^-53) of the reciprocal, and other
// than the IEEE quotient in the last bit of 0.06 % of the operands.  For normal
// numbers below 2^1022.
__device__ __forceinline__ double crcp(double a) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
  const double e = fma(-a, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// quotients; by the short reciprocal in the FP64 state (within 2 roundings)
__device__ __forceinline__ float quot(float a, float b) { return a / b; }
__device__ __forceinline__ double quot(double a, double b) { return a * crcp(b); }
// (1 / x)^(2/7), the Exner factor of x = p / p0, FP64: one step of the
// third-order iteration y (1 + e/7 + (4/49) e^2), e = 1 - x^2 y^7, on the FP32
// power (e below 6e-6; the next term, 0.06 e^3, is below 2e-17 of the result).
// A dozen multiply-adds in place of a quotient and a power, within 1.42
// roundings for 1e-6 <= x <= 1.3.
__device__ __forceinline__ double exner(double x) {
  const double y = (double)exp2f(-2.f / 7.f * log2f((float)x));
  const double y2 = y * y, y4 = y2 * y2, y7 = y4 * y2 * y;
  const double e = fma(-(x * x), y7, 1.0);
  return fma(y * e, fma(e, 4.0 / 49.0, 1.0 / 7.0), y);
}

// sum of c[k] w^k, k < N
template <typename R, int N>
__device__ __forceinline__ R series(const R* c, R w) {
  R v = c[N - 1];
#pragma unroll
  for (int k = N - 2; k >= 0; --k) v = v * w + c[k];
  return v;
}

// float to double with integer operations: the conversion instruction runs on
// the FP64 pipe (two lanes per clock and SM) and bounds a kernel that does
// little else.  The same result; zero, subnormal numbers, infinities and NaN
// take the instruction.  (Inside the FFT kernels of the eddy form it costs
// more registers than it saves: 4.5 -> 4.8 ms per T254L64 step.)
__device__ __forceinline__ double float_to_double(float x) {
  const uint32_t u = __float_as_uint(x), a = u & 0x7fffffffu;
  if (a - 0x00800000u >= 0x7f000000u) return (double)x;
  return __hiloint2double((int)((u & 0x80000000u) | ((a >> 3) + 0x38000000u)), (int)(u << 29));
}

// Copies a host array that may go away to the device, in the order of the
// stream whose kernels read it.  Not cudaMemcpy or cudaMemset: they run on the
// legacy default stream and may return before the device has the bytes, and
// the non-blocking streams used here do not wait for that stream.
inline void upload_on(void* dst, const void* src, size_t bytes, cudaStream_t s) {
  if (bytes == 0) return;
  GD_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
  GD_CUDA(cudaStreamSynchronize(s));
}

// Launch accounting (reported by gd_launch_count).
extern long long g_launches;
inline void count_launch(int n = 1) { g_launches += n; }

}  // namespace gd
