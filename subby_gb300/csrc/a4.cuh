// Length-4 vectors in packed FP32x2 form: the arithmetic of the A = 4 kernels
// (k_tree4.cu, k_inside4.cu), which agree bit for bit on the inside pass.
#pragma once
#include <cuda_runtime.h>

namespace subby {
namespace {

// what an outside pass writes (k_tree4.cu, k_pass4.cu)
constexpr int kOutSum = 0, kOutBranch = 1, kOutPost = 2;
constexpr double kLn2q = 0.69314718055994530942;

struct F4 {
  float2 a, b;
};

__device__ __forceinline__ F4 ld4s(const float *p) {
  const float4 t = *reinterpret_cast<const float4 *>(p);
  return F4{make_float2(t.x, t.y), make_float2(t.z, t.w)};
}
__device__ __forceinline__ F4 mul4(const F4 &x, const F4 &y) {
  return F4{__fmul2_rn(x.a, y.a), __fmul2_rn(x.b, y.b)};
}
__device__ __forceinline__ F4 scale4(const F4 &x, float s) {
  const float2 ss = make_float2(s, s);
  return F4{__fmul2_rn(x.a, ss), __fmul2_rn(x.b, ss)};
}
__device__ __forceinline__ F4 fma4(float s, const F4 &y, const F4 &z) {
  const float2 ss = make_float2(s, s);
  return F4{__ffma2_rn(ss, y.a, z.a), __ffma2_rn(ss, y.b, z.b)};
}
__device__ __forceinline__ float sum4(const F4 &x) { return (x.a.x + x.a.y) + (x.b.x + x.b.y); }
__device__ __forceinline__ float dot4(const F4 &x, const F4 &y) {
  const float2 t = __ffma2_rn(x.b, y.b, __fmul2_rn(x.a, y.a));
  return t.x + t.y;
}

// Multiply by 2^-e with e = floor(log2(max)); returns e.  The scale factor is
// built from the exponent field of the max, so zero / subnormal maxima take
// e = -127 (scale 2^127): still an exact power of two, no branch.
__device__ __forceinline__ int rescale4(F4 &u) {
  const float m = fmaxf(fmaxf(u.a.x, u.a.y), fmaxf(u.b.x, u.b.y));
  const int E = __float_as_int(m) >> 23;  // m >= 0: sign bit clear
  const float s = __int_as_float((254 - E) << 23);
  u = scale4(u, s);
  return E - 127;
}

// y = M u  with MT rows (MT[j][b] = M[b][j])
__device__ __forceinline__ F4 matvec4(const float *MTn, const F4 &u) {
  F4 y = scale4(ld4s(MTn), u.a.x);
  y = fma4(u.a.y, ld4s(MTn + 4), y);
  y = fma4(u.b.x, ld4s(MTn + 8), y);
  y = fma4(u.b.y, ld4s(MTn + 12), y);
  return y;
}
// y_a = sum_i d_i M[i][a] = dot(MT row a, d)
__device__ __forceinline__ F4 vecmat4(const float *MTn, const F4 &d) {
  return F4{make_float2(dot4(ld4s(MTn), d), dot4(ld4s(MTn + 4), d)),
            make_float2(dot4(ld4s(MTn + 8), d), dot4(ld4s(MTn + 12), d))};
}

__device__ __forceinline__ int tcode4(int tok) { return (int)min((unsigned)tok, 4u); }
__device__ __forceinline__ int tung4(int tok) { return (unsigned)tok <= 4u; }

}  // namespace
}  // namespace subby
