// Shared definitions for the GB300 2DTM kernels: status codes, complex helpers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/leopard_gb300.h"

namespace lgb {

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// a * conj(b)
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }

// float -> double with integer operations (exponent re-bias, mantissa shift):
// exact for normal floats, which leaves the FP64 pipe (about one operation per
// SM per clock on this GPU, conversions included) to the additions.  Zero,
// subnormal, inf and nan go through the converter.
__device__ __forceinline__ double f2d_bits(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned ex = (u >> 23) & 0xffu;
  if (ex == 0u || ex == 0xffu) return (double)f;
  const unsigned hi = (u & 0x80000000u) | ((ex + 896u) << 20) | ((u & 0x7fffffu) >> 3);
  return __hiloint2double((int)hi, (int)(u << 29));
}
// double -> float rounded to nearest even with integer operations, for values
// in the range of normal floats; the others go through the converter.
__device__ __forceinline__ float d2f_bits(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned ex = (hi >> 20) & 0x7ffu;
  if (ex < 897u || ex > 1149u) return (float)d;
  const unsigned f = ((ex - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
  const unsigned rest = lo << 3;  // the 29 bits below the float's mantissa
  const unsigned up = rest > 0x80000000u || (rest == 0x80000000u && (f & 1u));
  return __uint_as_float((hi & 0x80000000u) | (f + up));
}
// d = x + y to 48 bits with integer operations: x the leading 24 bits
// (truncated), y the rest.  For |d| < 2^128; below 2^-74 y is dropped, below
// 2^-126 both are zero.
__device__ __forceinline__ float2 d2f_split(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const int ex = (int)((hi >> 20) & 0x7ffu);
  const unsigned sign = hi & 0x80000000u;
  if (ex < 897) return make_float2(0.f, 0.f);
  const float x = __uint_as_float(sign | ((unsigned)(ex - 896) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
  const int ey = ex - 948;  // biased exponent of 2^(ex - 1023 - 52)
  const float unit = ey > 0 ? __uint_as_float(sign | ((unsigned)ey << 23)) : 0.f;
  return make_float2(x, (float)(lo & 0x1fffffffu) * unit);
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// the same as one packed multiply (an issue slot less, the same rounding)
__device__ __forceinline__ float2 cscale_packed(float2 a, float s) {
  float2 r;
  asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %4};\n mul.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(s));
  return r;
}
// multiply by DIR*i  (DIR = +1: i, DIR = -1: -i)
template <int DIR>
__device__ __forceinline__ float2 mul_i(float2 a) {
  return DIR > 0 ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// ---- async copy helpers (16-byte cp.async, completion via wait_group) -------
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Status codes returned by every C-ABI entry point (see include/leopard_gb300.h).
#define LGB_CUDA_TRY(expr)                                   \
  do {                                                       \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess) return LGB_ERR_CUDA;              \
  } while (0)

}  // namespace lgb
