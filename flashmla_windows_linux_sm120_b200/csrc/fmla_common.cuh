// Shared device helpers for the sm_100a attention kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fmla {

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// 16-byte asynchronous global->shared copy; when !valid the destination is
// zero-filled and the source is not read.
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int sz = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(sz) : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// 32 bytes to global memory: one 256-bit store when the address allows it, else two 128-bit stores
__device__ __forceinline__ void st_global_32B(void* p, const uint32_t (&w)[8]) {
  if ((reinterpret_cast<uintptr_t>(p) & 31u) == 0) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]),
                 "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  } else {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// Named barrier over `nthreads` threads (ids 1..15; 0 is __syncthreads).
__device__ __forceinline__ void bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(nthreads) : "memory");
}

__device__ __forceinline__ uint32_t pack_f16x2(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// two floats -> one 32-bit word of the 16-bit output type (bf16, or fp16 when F16)
template <bool F16>
__device__ __forceinline__ uint32_t pack_16x2(float lo, float hi) {
  if constexpr (F16) return pack_f16x2(lo, hi);
  else return pack_bf16x2(lo, hi);
}
// Programmatic dependent launch: a kernel launched with the programmatic-stream-serialization attribute may start
// (prologue, resident and waiting) while its predecessor in the stream still runs; pdl_wait() blocks until the
// predecessor has completed and its memory is visible, pdl_allow_dependents() lets the successor start early.
// Both are no-ops for plain launches.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_allow_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

__device__ __forceinline__ float neg_inf() { return __int_as_float(0xff800000); }
__device__ __forceinline__ float pos_inf() { return __int_as_float(0x7f800000); }

// Two floats at a time (one instruction each).
struct F2 {
  float lo, hi;
};
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 d;
  asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\nfma.rn.f32x2 d, a, b, c;\nmov.b64 {%0, %1}, d;\n}\n"
      : "=f"(d.lo), "=f"(d.hi)
      : "f"(a.lo), "f"(a.hi), "f"(b.lo), "f"(b.hi), "f"(c.lo), "f"(c.hi));
  return d;
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 d;
  asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nadd.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}\n"
      : "=f"(d.lo), "=f"(d.hi)
      : "f"(a.lo), "f"(a.hi), "f"(b.lo), "f"(b.hi));
  return d;
}
__device__ __forceinline__ F2 f2(float x) { return F2{x, x}; }
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 d;
  asm("{\n.reg .b64 a, b, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmul.rn.f32x2 d, a, b;\nmov.b64 {%0, %1}, d;\n}\n"
      : "=f"(d.lo), "=f"(d.hi)
      : "f"(a.lo), "f"(a.hi), "f"(b.lo), "f"(b.hi));
  return d;
}
// 2^x for -127 <= x <= 128 on the multiply-add pipe: x = n + f with n the nearest whole number (held in the low bits of x + 1.5 * 2^23)
// and |f| <= 1/2, and 2^f = 1 + f q(f) with the polynomial of least largest relative error (fitted with Lawson's weights: 1.1e-7, in
// fp32 1.7e-7 over the range; the special function unit's 2^x is specified to 2.4e-7).  At the ends exactly 0 and infinity; beyond
// them the sum of the exponents would wrap into the sign.  tests/test_gpu_exp2.py
__device__ __forceinline__ F2 f2_exp2_inside(F2 x) {
  const F2 t = f2_add(x, f2(12582912.f));
  const F2 n = f2_add(t, f2(-12582912.f));
  const F2 f = f2_fma(n, f2(-1.f), x);
  F2 r = f2_fma(f, f2(0x1.5bba14p-10f), f2(0x1.3cea88p-7f));
  r = f2_fma(r, f, f2(0x1.c6b752p-5f));
  r = f2_fma(r, f, f2(0x1.ebf9bcp-3f));
  r = f2_fma(r, f, f2(0x1.62e42ap-1f));
  r = f2_fma(r, f, f2(1.f));
  r.lo = __uint_as_float(__float_as_uint(r.lo) + (__float_as_uint(t.lo) << 23));
  r.hi = __uint_as_float(__float_as_uint(r.hi) + (__float_as_uint(t.hi) << 23));
  return r;
}
// 2^x for x <= 128, 0 for NaN
__device__ __forceinline__ F2 f2_exp2_to_128(F2 x) {
  x.lo = fmaxf(x.lo, -127.f);
  x.hi = fmaxf(x.hi, -127.f);
  return f2_exp2_inside(x);
}
// 2^x for every x, NaN for NaN
__device__ __forceinline__ F2 f2_exp2(F2 x) {
  const auto inside = [](float v) {
    asm("{\n.reg .f32 t;\nmax.NaN.f32 t, %0, 0fC2FE0000;\nmin.NaN.f32 %0, t, 0f43000000;\n}\n" : "+f"(v));      // -127, 128
    return v;
  };
  x.lo = inside(x.lo);
  x.hi = inside(x.hi);
  return f2_fma(x, f2(0.f), f2_exp2_inside(x));
}
// the largest of three (NaN only if all are)
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

}  // namespace fmla
