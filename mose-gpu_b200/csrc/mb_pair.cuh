// mb_pair.cuh -- two values of the flux arithmetic type that travel together: in FP32 a 64-bit register pair, on which
// sm_100 adds, multiplies and fuses both halves with one instruction (.f32x2, each half rounded to nearest, subnormals
// flushed as in the scalar code of these units); in FP64 two scalars.
#pragma once

namespace mb {

template <typename R> struct V2;
template <> struct __align__(16) V2<double> { double x, y; };
template <> struct __align__(8) V2<float> { unsigned long long q; };

template <typename R> __device__ __forceinline__ V2<R> mk2(R x, R y);
template <> __device__ __forceinline__ V2<double> mk2(double x, double y) { return V2<double>{x, y}; }
template <> __device__ __forceinline__ V2<float> mk2(float x, float y) {
  V2<float> r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.q) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ double lo2(const V2<double>& a) { return a.x; }
__device__ __forceinline__ double hi2(const V2<double>& a) { return a.y; }
__device__ __forceinline__ float lo2(const V2<float>& a) {
  float x;
  asm("{\n .reg .b32 t;\n mov.b64 {%0, t}, %1;\n}" : "=f"(x) : "l"(a.q));
  return x;
}
__device__ __forceinline__ float hi2(const V2<float>& a) {
  float y;
  asm("{\n .reg .b32 t;\n mov.b64 {t, %0}, %1;\n}" : "=f"(y) : "l"(a.q));
  return y;
}
template <typename R> __device__ __forceinline__ V2<R> dup2(R x) { return mk2<R>(x, x); }
__device__ __forceinline__ V2<double> operator+(V2<double> a, V2<double> b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ V2<double> operator-(V2<double> a, V2<double> b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ V2<double> operator*(V2<double> a, V2<double> b) { return {a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ V2<double> fma2(V2<double> a, V2<double> b, V2<double> c) {
  return {fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)};
}
__device__ __forceinline__ V2<float> operator+(V2<float> a, V2<float> b) {
  V2<float> r;
  asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.q) : "l"(a.q), "l"(b.q));
  return r;
}
__device__ __forceinline__ V2<float> operator-(V2<float> a, V2<float> b) {
  V2<float> r;
  asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.q) : "l"(a.q), "l"(b.q));
  return r;
}
__device__ __forceinline__ V2<float> operator*(V2<float> a, V2<float> b) {
  V2<float> r;
  asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.q) : "l"(a.q), "l"(b.q));
  return r;
}
__device__ __forceinline__ V2<float> fma2(V2<float> a, V2<float> b, V2<float> c) {
  V2<float> r;
  asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.q) : "l"(a.q), "l"(b.q), "l"(c.q));
  return r;
}

// reciprocal of the flux path. In FP32 within 1 ulp, 0 for |x| > 2^126 (the result would be subnormal) and infinite below
// 2^-126. No denominator of the path comes near either end before the terms beside it overflow: densities are at least
// 1e-20, the smallest sums carry 1e-30, and van Albada's squares reach 2^126 at slopes of 9e18, where its cubes have been
// infinite since 7e12.
__device__ __forceinline__ double rcp_(double x) { return 1.0 / x; }
__device__ __forceinline__ float rcp_(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

}  // namespace mb
