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

constexpr int kQuantThreads = 256, kQuantUnroll = 2;

__device__ __forceinline__ void load256_stream(const uint8_t* p, uint32_t* v) {
  asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "l"(p));
}
// Half a block, 16 consecutive elements, as fp32.  WIDE: 32-byte loads (the input starts on a 32-byte boundary).
template <class T, bool WIDE>
struct Load16 {
  static constexpr int kWords = 16 * (int)sizeof(typename T::elem) / 4;
  uint32_t v[kWords];
  __device__ __forceinline__ void load(const uint8_t* p) {
    if constexpr (WIDE) {
#pragma unroll
      for (int i = 0; i < kWords / 8; ++i) load256_stream(p + 32 * i, v + 8 * i);
    } else {
#pragma unroll
      for (int i = 0; i < kWords / 4; ++i) {
        const u128 t = load128_stream(p + 16 * i);
        v[4 * i] = (uint32_t)t.x;
        v[4 * i + 1] = (uint32_t)(t.x >> 32);
        v[4 * i + 2] = (uint32_t)t.y;
        v[4 * i + 3] = (uint32_t)(t.y >> 32);
      }
    }
  }
  __device__ __forceinline__ void get(float* f) const {
#pragma unroll
    for (int i = 0; i < kWords / 2; ++i) T::unpack((uint64_t)v[2 * i] | ((uint64_t)v[2 * i + 1] << 32), f + i * T::kPer64);
  }
};

// What converting to e4m3fn gives without saturation: NaN (with the sign) from halfway past 448 on.
__device__ __forceinline__ uint8_t e4m3_nosat(float q) {
  if (!(fabsf(q) <= 464.f)) return (uint8_t)(0x7fu | ((__float_as_uint(q) >> 24) & 0x80u));
  return float_to_e4m3(q);
}

// Bound by HBM: 3 bytes and a bit per bf16 element; 8192 x 4096 takes 18.5 us on fixed buffers (5.4 TB/s).  Two lanes share a block of 32:
// 32-byte loads, 16-byte stores, one shuffle for the block maximum.  (Four lanes with 16-byte loads and 8-byte stores
// took 22 - 25 us whatever the unrolling and the grid.)  The maximum is taken on the bit patterns, where NaN is larger
// than everything, as amax has it.  The chain of torch kernels this replaces made about a dozen passes over fp32
// copies: a linear layer of 8192 x 4096 -> 1792 (quantise, tile, GEMM) took 640 us.
template <class T, bool WIDE>
__global__ void __launch_bounds__(kQuantThreads) mx_quant_kernel(const uint8_t* __restrict__ x, uint8_t* __restrict__ data,
                                                                 uint8_t* __restrict__ scale, uint64_t nhalves) {
  constexpr int kBytes = 16 * (int)sizeof(typename T::elem);
  const uint64_t base = (uint64_t)blockIdx.x * (kQuantThreads * kQuantUnroll) + threadIdx.x;
  Load16<T, WIDE> in[kQuantUnroll];
#pragma unroll
  for (int u = 0; u < kQuantUnroll; ++u) {
    const uint64_t g = base + u * kQuantThreads;
    if (g < nhalves) in[u].load(x + g * kBytes);
  }
#pragma unroll
  for (int u = 0; u < kQuantUnroll; ++u) {
    // nhalves is even: the two lanes of a block are in or out together
    const uint64_t g = base + u * kQuantThreads;
    const bool live = g < nhalves;
    float f[16];
    uint32_t m = 0;
    if (live) {
      in[u].get(f);
#pragma unroll
      for (int i = 0; i < 16; ++i) m = max(m, __float_as_uint(f[i]) & 0x7fffffffu);
    }
    m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
    if (!live) continue;
    // smallest power of two 2^(e - 127) with amax <= 448 * 2^(e - 127): from the exponent, one more past 1.75 * 2^k
    uint32_t e = 127 - 8;
    if (m >= 0x7f800000u) e = ue8m0_for_amax(__uint_as_float(m));
    else if (m != 0) e = (uint32_t)max((int)(m >> 23) - 8 + ((m & 0x7fffffu) > 0x600000u ? 1 : 0), 1);
    const float inv = __uint_as_float(e == 254u ? 0x00400000u : (254u - e) << 23);   // 2^(127 - e): exact
    uint32_t w[4] = {0, 0, 0, 0};
    if (m < 0x7f800000u) {   // every quotient is at most 448: nothing saturates
#pragma unroll
      for (int i = 0; i < 8; ++i)
        w[i >> 1] |= (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(f[2 * i] * inv, f[2 * i + 1] * inv), __NV_SATFINITE, __NV_E4M3)
                     << (16 * (i & 1));
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) w[i >> 2] |= (uint32_t)e4m3_nosat(f[i] * inv) << (8 * (i & 3));
    }
    *reinterpret_cast<uint4*>(data + g * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    if ((threadIdx.x & 1) == 0) scale[g >> 1] = (uint8_t)e;
  }
}

// Scales [rows, kq] of 4-byte words (four blocks along K) -> [rows / 128][kq][32][4] words: word (r % 32, (r % 128) / 32)
// of an atom.  One CTA takes 128 rows x 8 words through shared memory: whole sectors on the reading side, whole lines on
// the writing side, all loads of a thread in flight, and enough CTAs (8192 x 4096 has 256) that the one round trip is all
// that is left.
constexpr int kTileWords = 8;
__global__ void __launch_bounds__(256) mx_tile_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, uint32_t kq) {
  __shared__ uint32_t s[128][kTileWords + 1];
  const uint32_t R = blockIdx.y, k0 = blockIdx.x * kTileWords;
  const uint32_t nk = min((uint32_t)kTileWords, kq - k0);
  uint32_t v[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t r = j * 32 + (threadIdx.x >> 3), k = threadIdx.x & 7;
    if (k < nk) v[j] = in[((uint64_t)R * 128 + r) * kq + k0 + k];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j * 32 + (threadIdx.x >> 3)][threadIdx.x & 7] = v[j];
  __syncthreads();
  uint32_t* o = out + ((uint64_t)R * kq + k0) * 128;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t i = j * 256 + threadIdx.x, w = i & 127;   // word of the atom
    if (i < nk * 128) o[i] = s[(w & 3) * 32 + (w >> 2)][i >> 7];
  }
}

template <class T>
static void go_quant(const void* x, void* data, void* scale, uint64_t nelems, cudaStream_t s) {
  const uint64_t halves = nelems / 16, chunk = (uint64_t)kQuantThreads * kQuantUnroll;
  const unsigned grid = (unsigned)((halves + chunk - 1) / chunk);
  if (((uintptr_t)x & 31) == 0)
    mx_quant_kernel<T, true><<<grid, kQuantThreads, 0, s>>>((const uint8_t*)x, (uint8_t*)data, (uint8_t*)scale, halves);
  else
    mx_quant_kernel<T, false><<<grid, kQuantThreads, 0, s>>>((const uint8_t*)x, (uint8_t*)data, (uint8_t*)scale, halves);
}

cudaError_t launch_mx_quant(int dtype, const void* x, void* data, void* scale, uint64_t nelems, cudaStream_t s) {
  if (nelems / 16 / (kQuantThreads * kQuantUnroll) >= 0x7fffffffull) return cudaErrorInvalidValue;
  count_launch();
  switch (dtype) {
    case DT_F32: go_quant<F32>(x, data, scale, nelems, s); break;
    case DT_F16: go_quant<F16>(x, data, scale, nelems, s); break;
    case DT_BF16: go_quant<BF16>(x, data, scale, nelems, s); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_mx_tile(const void* in, void* out, uint32_t row_blocks, uint32_t kq, cudaStream_t s) {
  count_launch();
  mx_tile_kernel<<<dim3((kq + kTileWords - 1) / kTileWords, row_blocks), 256, 0, s>>>((const uint32_t*)in, (uint32_t*)out, kq);
  return cudaGetLastError();
}

}  // namespace mt
