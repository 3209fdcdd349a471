// Complex helpers and constants of the FP32 transforms (gb_fft.cu, gb_rows.cu).
#pragma once

#include <cuda_runtime.h>

namespace gb {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float c, float s) {
  return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
}
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }
// both parts in one packed instruction (a negated operand costs nothing)
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return __fadd2_rn(a, make_float2(-b.x, -b.y));
}
// a + s i b, a - s i b: two scalar sums, as the packed form would first swap b's parts
template <int S> __device__ __forceinline__ float2 cadd_si(float2 a, float2 b) {
  return S > 0 ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, a.y - b.x);
}
template <int S> __device__ __forceinline__ float2 csub_si(float2 a, float2 b) {
  return cadd_si<-S>(a, b);
}
// a * (s i)
template <int S> __device__ __forceinline__ float2 mul_si(float2 a) {
  return S > 0 ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

constexpr float kR2 = 0.70710678118654752f;  // cos(pi/4)
constexpr float kC8 = 0.92387953251128674f;  // cos(pi/8)
constexpr float kS8 = 0.38268343236508977f;  // sin(pi/8)

// cos / sin(2 pi k / 32), k < 16
static __device__ __constant__ float kCos32[16] = {1.0f, 0.98078528040323043f, 0.92387953251128674f, 0.83146961230254524f, 0.70710678118654757f, 0.55557023301960229f, 0.38268343236508984f, 0.19509032201612833f, 0.0f, -0.19509032201612819f, -0.38268343236508973f, -0.55557023301960196f, -0.70710678118654746f, -0.83146961230254535f, -0.92387953251128674f, -0.98078528040323043f};
static __device__ __constant__ float kSin32[16] = {0.0f, 0.19509032201612825f, 0.38268343236508978f, 0.55557023301960218f, 0.70710678118654746f, 0.83146961230254524f, 0.92387953251128674f, 0.98078528040323043f, 1.0f, 0.98078528040323043f, 0.92387953251128674f, 0.83146961230254546f, 0.70710678118654757f, 0.55557023301960218f, 0.38268343236508989f, 0.19509032201612861f};

}  // namespace gb
