// FP8 KV-cache writer: bf16 [num_tokens, 576] -> 656-byte token records
// (512 x e4m3 | 4 x fp32 scale | 64 x bf16 rope; README.md:162-170).
// Arithmetic of tests/quant.py:3-35: per 128-wide tile, scale = bf16(amax/448)
// widened to fp32, q = e4m3_rn(fp32(x) / scale).  One warp per token.
// Bound by HBM (1 812 bytes per token) once the quotients leave it to be: with sixteen IEEE divisions per lane 60 000 tokens took 30.1 us
// on the device (3.6 TB/s), 25 000 10.7, 8 192 4.9; now 21.3 (5.1 TB/s), 7.7 and 3.9.  (A call of 8 192 takes 6.1 us either way: the host.)
#include "fmla_common.cuh"
#include "kernels.h"

#include <cuda_fp8.h>

namespace fmla {

// x / b rounded to nearest, from y = 1 / b rounded to nearest: the product x y and one correction step by its exact remainder
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).  That the result is the rounded
// quotient was checked in exact arithmetic for all pairs of bf16 significands, which is all there is to x and b; kDivLo and
// kDivHi keep the remainder and the products clear of underflow and overflow for every quotient that does not round to zero
// (2^-10 is half the smallest e4m3 number).  The sign is that of x: the correction would turn -0 into +0.
constexpr float kDivLo = 0x1p-80f, kDivHi = 0x1p100f;
__device__ __forceinline__ float divide_by(float x, float b, float y) {
  const float q = x * y;
  return copysignf(fmaf(fmaf(-b, q, x), y, q), x);
}

__global__ void __launch_bounds__(256) quantize_kv_fp8_kernel(const __nv_bfloat16* __restrict__ kv, int64_t kv_stride_row,
                                                             int num_tokens, const int* __restrict__ dst_slots,
                                                             unsigned char* __restrict__ cache, int64_t cache_stride_slot) {
  const int tok = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (tok >= num_tokens) return;
  const int slot = dst_slots ? dst_slots[tok] : tok;
  const __nv_bfloat16* src = kv + (int64_t)tok * kv_stride_row;
  unsigned char* rec = cache + (int64_t)slot * cache_stride_slot;

  // The row is asked for before the slot is looked at (a skipped token's row is there all the same).  Of 8 192 tokens all, half, one in
  // twenty or none with a slot 6.4 -> 4.6 us, 4.9 -> 3.4, 2.8 -> 2.4 and 1.6 -> 1.9; of 256 2.6 -> 2.0, 2.5 -> 2.0, 2.4 -> 1.8 and 1.2 -> 1.4 (sixteen
  // divisions and the slot first -> this): only a call in which no token has a slot loses.
  uint4 raw[2], rope = make_uint4(0, 0, 0, 0);
  raw[0] = *reinterpret_cast<const uint4*>(src + lane * 16);
  raw[1] = *reinterpret_cast<const uint4*>(src + lane * 16 + 8);
  if (lane < 8) rope = *reinterpret_cast<const uint4*>(src + 512 + lane * 8);
  if (slot < 0) return;
  float x[16];
  const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(raw);
  float amax = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 f = __bfloat1622float2(h2[i]);
    x[2 * i] = f.x;
    x[2 * i + 1] = f.y;
    amax = fmaxf(amax, fmaxf(fabsf(f.x), fabsf(f.y)));
  }
#pragma unroll
  for (int off = 1; off <= 4; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  const float scale = __bfloat162float(__float2bfloat16_rn(__fdiv_rn(amax, 448.0f)));
  if (scale >= kDivLo && scale <= kDivHi) {
    const float y = __frcp_rn(scale);
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = divide_by(x[i], scale, y);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = __fdiv_rn(x[i], scale);
  }
  uint32_t q[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(x[i * 4], x[i * 4 + 1]), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(x[i * 4 + 2], x[i * 4 + 3]), __NV_SATFINITE, __NV_E4M3);
    q[i] = lo | hi << 16;
  }
  *reinterpret_cast<uint4*>(rec + lane * 16) = make_uint4(q[0], q[1], q[2], q[3]);
  const float s_tile = __shfl_sync(0xffffffffu, scale, (lane & 3) * 8);
  if (lane < 4) reinterpret_cast<float*>(rec + 512)[lane] = s_tile;
  if (lane < 8) *reinterpret_cast<uint4*>(rec + 528 + lane * 16) = rope;
}

cudaError_t launch_quantize_kv_fp8(const void* kv, int64_t kv_stride_row, int num_tokens, const int* dst_slots, void* cache,
                                   int64_t cache_stride_slot, cudaStream_t stream) {
  if (num_tokens == 0) return cudaSuccess;
  quantize_kv_fp8_kernel<<<(num_tokens + 7) / 8, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(kv), kv_stride_row,
                                                                  num_tokens, dst_slots,
                                                                  reinterpret_cast<unsigned char*>(cache), cache_stride_slot);
  return cudaGetLastError();
}

}  // namespace fmla
