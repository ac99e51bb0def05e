// Block-scaled fp8 (MXFP8: e4m3 payload, one ue8m0 scale per 32 elements) sum over ranks.
//
// Every rank holds a quantised tensor (payload bytes + scale bytes) in the symmetric heap.  The sum is
// formed in one hop: the owner of a 32-element block reads that block and its scale from every rank,
// dequantises, accumulates in fp32 in rank order (bit-identical on every rank), picks the new block scale
// from the block's largest magnitude and quantises once.  Intermediate hops of a ring would requantise
// n - 1 times; here precision is lost exactly once.  all-reduce writes the result to every rank
// (two-shot), reduce-scatter keeps the owner's shard.
//
// The reference only sums fp16 (primitive.py:230-247); fp8 is on its roadmap (README.md:58-60).
#include "../device/prims.cuh"
#include "../device/reduce_ops.cuh"
#include "../device/sched.h"
#include "launch.h"
#include "mxfp8.h"

namespace mt {

constexpr int kMxThreads = 512;

// acc[0 .. 15] += the 16 e4m3 values of a half block times its scale
__device__ __forceinline__ void mx_accumulate(float* acc, u128 d, uint8_t sc) {
  const float s = ue8m0_to_float(sc);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint64_t w = k < 4 ? d.x : d.y;
    const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> (16 * (k & 3))), __NV_E4M3);
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    acc[2 * k] += f.x * s;
    acc[2 * k + 1] += f.y * s;
  }
}

// Blocks [lo, hi) of rank `me`: two lanes per block of 32.  Bound by the bytes in flight: with one lane per block, 256
// threads and one rank's loads at a time, 8 emulated ranks of 16 Mi elements took 131 us (2.1 TB/s); 65 us now.  Every load is a
// whole 512-byte line group per warp, the loads of all ranks (NR > 0: known at compile time) are issued before the first
// is used, and e4m3 is converted two at a time.
template <int NR>
__device__ __forceinline__ void mx_reduce_range(const MtDevComm& c, const Mxfp8Args& a, int lr, uint64_t lo, uint64_t hi) {
  const int n = NR > 0 ? NR : c.nranks, me = c.rank, half = threadIdx.x & 1;
  // every lane of a warp runs the same number of rounds: the two lanes of a block exchange their maxima
  for (uint64_t base = lo; base < hi; base += kMxThreads / 2) {
    const uint64_t b = base + (threadIdx.x >> 1);
    const bool live = b < hi;
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    if (live) {
      const uint64_t off = a.data_in_off + b * 32 + half * 16;
      if constexpr (NR > 0) {
        u128 d[NR];
        uint8_t sc[NR];
#pragma unroll
        for (int p = 0; p < NR; ++p) {
          d[p] = load128_relaxed_sys(c.heap[p] + off);
          sc[p] = *reinterpret_cast<const volatile uint8_t*>(c.heap[p] + a.scale_in_off + b);
        }
#pragma unroll
        for (int p = 0; p < NR; ++p) mx_accumulate(acc, d[p], sc[p]);
      } else {
        for (int p = 0; p < n; ++p) {
          const u128 d = load128_relaxed_sys(c.heap[p] + off);
          mx_accumulate(acc, d, *reinterpret_cast<const volatile uint8_t*>(c.heap[p] + a.scale_in_off + b));
        }
      }
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(acc[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    if (!live) continue;
    const uint8_t so = ue8m0_for_amax(amax);
    const float inv = 1.0f / ue8m0_to_float(so);
    u128 o = {0, 0};
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint64_t q = __nv_cvt_float2_to_fp8x2(make_float2(acc[2 * k] * inv, acc[2 * k + 1] * inv), __NV_SATFINITE, __NV_E4M3);
      if (k < 4) o.x |= q << (16 * k);
      else o.y |= q << (16 * (k - 4));
    }
    if (a.op == MX_ALLREDUCE) {
      for (int d = 0; d < n; ++d) {
        const int p = (me + d) % n;
        store128_relaxed_sys(c.heap[p] + a.data_out_off + b * 32 + half * 16, o);
        if (half == 0) *reinterpret_cast<volatile uint8_t*>(c.heap[p] + a.scale_out_off + b) = so;
      }
    } else {
      const uint64_t bl = b - (uint64_t)me * (a.nblocks / n);
      *reinterpret_cast<u128*>((uint8_t*)a.data_out[lr] + bl * 32 + half * 16) = o;
      if (half == 0) ((uint8_t*)a.scale_out[lr])[bl] = so;
    }
  }
}

__global__ void __launch_bounds__(kMxThreads, 1) mxfp8_kernel(const MtDevComm* comms, Mxfp8Args a) {
  __shared__ int s_fail;
  const int lr = blockIdx.y;
  const MtDevComm& c = comms[lr];
  const int n = c.nranks, me = c.rank;
  if (!rank_barrier(c, blockIdx.x, &s_fail)) return;
  // blocks this CTA works on, and inside them the ones this rank owns
  uint64_t lo, hi;
  if (a.op == MX_ALLREDUCE) {
    const MtRange r = mt_split(a.nblocks, gridDim.x, blockIdx.x, 1);
    const MtRange s = mt_split(r.hi - r.lo, n, me, 1);
    lo = r.lo + s.lo;
    hi = r.lo + s.hi;
  } else {
    const uint64_t per = a.nblocks / n;  // blocks per shard
    const MtRange r = mt_split(per, gridDim.x, blockIdx.x, 1);
    lo = (uint64_t)me * per + r.lo;
    hi = (uint64_t)me * per + r.hi;
  }
  switch (n) {
    case 2: mx_reduce_range<2>(c, a, lr, lo, hi); break;
    case 4: mx_reduce_range<4>(c, a, lr, lo, hi); break;
    case 8: mx_reduce_range<8>(c, a, lr, lo, hi); break;
    default: mx_reduce_range<0>(c, a, lr, lo, hi); break;
  }
  rank_barrier(c, blockIdx.x, &s_fail);
}

cudaError_t launch_mxfp8(const MtDevComm* comms, const Mxfp8Args& a, int nctas, int nlocal, cudaStream_t s) {
  Mxfp8Args args = a;
  void* p[] = {(void*)&comms, (void*)&args};
  return launch_any((const void*)mxfp8_kernel, dim3(nctas, nlocal), dim3(kMxThreads), p, s, nlocal > 1);
}

}  // namespace mt
