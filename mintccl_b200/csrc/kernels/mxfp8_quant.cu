// MXFP8 encoding: fp32 / fp16 / bf16 -> e4m3 payload with one ue8m0 scale per 32 elements, and the reordering of
// row-major scales into the layout tcgen05 reads.  Both give, bit for bit, what the torch expressions in
// ops/mxfp8.py give (which stay as the oracle and as the CPU path).
//
// The reference has no fp8 path; it is on its roadmap (README.md:58-60).
#include <cuda_runtime.h>
#include <stdint.h>

#include "../device/prims.cuh"
#include "../device/reduce_ops.cuh"
#include "launch.h"
#include "mxfp8.h"

namespace mt {

constexpr int kQuantThreads = 256, kQuantUnroll = 4;

// Eight consecutive elements as fp32.
template <class T>
struct Load8 {
  static constexpr int kBytes = 16;
  u128 v;
  __device__ __forceinline__ void load(const uint8_t* p) { v = load128_stream(p); }
  __device__ __forceinline__ void get(float* f) const {
    T::unpack(v.x, f);
    T::unpack(v.y, f + 4);
  }
};
template <>
struct Load8<F32> {
  static constexpr int kBytes = 32;
  u128 a, b;
  __device__ __forceinline__ void load(const uint8_t* p) {
    a = load128_stream(p);
    b = load128_stream(p + 16);
  }
  __device__ __forceinline__ void get(float* f) const {
    F32::unpack(a.x, f);
    F32::unpack(a.y, f + 2);
    F32::unpack(b.x, f + 4);
    F32::unpack(b.y, f + 6);
  }
};

// What converting to e4m3fn gives without saturation: NaN (with the sign) from halfway past 448 on.
__device__ __forceinline__ uint8_t e4m3_nosat(float q) {
  if (!(fabsf(q) <= 464.f)) return (uint8_t)(0x7fu | ((__float_as_uint(q) >> 24) & 0x80u));
  return float_to_e4m3(q);
}

// Bound by HBM: 3 bytes and a bit per bf16 element.  Four lanes share a block of 32 (8 elements each: 16-byte loads,
// 8-byte stores, two shuffles for the block maximum), four groups per thread are in flight; the maximum is taken on
// the bit patterns, where NaN is larger than everything, as amax has it.  The chain of torch kernels this replaces
// made about a dozen passes over fp32 copies.  A linear layer of 8192 x 4096 -> 1792 (quantise, tile, GEMM) went from
// 640 to 97 us with the two kernels of this file; the GEMM is 65 of them.
template <class T>
__global__ void __launch_bounds__(kQuantThreads) mx_quant_kernel(const uint8_t* __restrict__ x, uint8_t* __restrict__ data,
                                                                 uint8_t* __restrict__ scale, uint64_t ngroups) {
  constexpr uint64_t kChunk = (uint64_t)kQuantThreads * kQuantUnroll;
  for (uint64_t base = (uint64_t)blockIdx.x * kChunk; base < ngroups; base += (uint64_t)gridDim.x * kChunk) {
    Load8<T> in[kQuantUnroll];
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) {
      const uint64_t g = base + u * kQuantThreads + threadIdx.x;
      if (g < ngroups) in[u].load(x + g * Load8<T>::kBytes);
    }
#pragma unroll
    for (int u = 0; u < kQuantUnroll; ++u) {
      // ngroups is a multiple of 4: the four lanes of a block are in or out together
      const uint64_t g = base + u * kQuantThreads + threadIdx.x;
      const bool live = g < ngroups;
      float f[8];
      uint32_t m = 0;
      if (live) {
        in[u].get(f);
#pragma unroll
        for (int i = 0; i < 8; ++i) m = max(m, __float_as_uint(f[i]) & 0x7fffffffu);
      }
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
      if (!live) continue;
      const uint32_t e = ue8m0_for_amax(__uint_as_float(m));
      const float inv = __uint_as_float(e == 254u ? 0x00400000u : (254u - e) << 23);   // 2^(127 - e): exact
      uint64_t w = 0;
      if (m < 0x7f800000u) {   // every quotient is at most 448: nothing saturates
#pragma unroll
        for (int i = 0; i < 4; ++i)
          w |= (uint64_t)__nv_cvt_float2_to_fp8x2(make_float2(f[2 * i] * inv, f[2 * i + 1] * inv), __NV_SATFINITE, __NV_E4M3)
               << (16 * i);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) w |= (uint64_t)e4m3_nosat(f[i] * inv) << (8 * i);
      }
      *reinterpret_cast<uint64_t*>(data + g * 8) = w;
      if ((threadIdx.x & 3) == 0) scale[g >> 2] = (uint8_t)e;
    }
  }
}

// Scales [rows, kq] of 4-byte words (four blocks along K) -> [rows / 128][kq][32][4] words: word (r % 32, (r % 128) / 32)
// of an atom.  One CTA takes 128 rows x 32 words through shared memory, so that both sides are whole lines.
__global__ void __launch_bounds__(256) mx_tile_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t kq) {
  __shared__ uint32_t s[128][33];
  const uint32_t R = blockIdx.y, k0 = blockIdx.x * 32;
  const uint32_t nk = min(32u, kq - k0);
  for (uint32_t i = threadIdx.x; i < 128 * 32; i += 256) {
    const uint32_t r = i >> 5, k = i & 31;
    if (k < nk) s[r][k] = in[((uint64_t)R * 128 + r) * kq + k0 + k];
  }
  __syncthreads();
  uint32_t* o = out + ((uint64_t)R * kq + k0) * 128;
  for (uint32_t i = threadIdx.x; i < nk * 128; i += 256) {
    const uint32_t w = i & 127;   // word of the atom
    o[i] = s[(w & 3) * 32 + (w >> 2)][i >> 7];
  }
}

cudaError_t launch_mx_quant(int dtype, const void* x, void* data, void* scale, uint64_t nelems, int sms, cudaStream_t s) {
  const uint64_t groups = nelems / 8, chunk = (uint64_t)kQuantThreads * kQuantUnroll;
  uint64_t grid = (groups + chunk - 1) / chunk;
  if (grid > (uint64_t)sms * 8) grid = (uint64_t)sms * 8;
  const uint8_t* p = (const uint8_t*)x;
  count_launch();
  switch (dtype) {
    case DT_F32: mx_quant_kernel<F32><<<(unsigned)grid, kQuantThreads, 0, s>>>(p, (uint8_t*)data, (uint8_t*)scale, groups); break;
    case DT_F16: mx_quant_kernel<F16><<<(unsigned)grid, kQuantThreads, 0, s>>>(p, (uint8_t*)data, (uint8_t*)scale, groups); break;
    case DT_BF16: mx_quant_kernel<BF16><<<(unsigned)grid, kQuantThreads, 0, s>>>(p, (uint8_t*)data, (uint8_t*)scale, groups); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_mx_tile(const void* in, void* out, uint32_t row_blocks, uint32_t kq, cudaStream_t s) {
  count_launch();
  mx_tile_kernel<<<dim3((kq + 31) / 32, row_blocks), 256, 0, s>>>((const uint32_t*)in, (uint32_t*)out, kq);
  return cudaGetLastError();
}

}  // namespace mt
