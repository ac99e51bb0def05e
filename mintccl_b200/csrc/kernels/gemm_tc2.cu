// GEMM on CTA pairs: C[M, N] = A[M, K] * B[N, K]^T with tcgen05.mma.cta_group::2.
//
// Two CTAs of one cluster (neighbouring SMs) compute one tile of 256 rows and 256, 224, 128 or 64 columns (the widths:
// see gemm_pair_kernel).  Each CTA stages 128 rows of A and half the tile's rows of B per K block, so the tensor cores of
// both SMs read every B row from ONE shared memory only: at 256 columns, per SM and MMA, the shared-memory traffic (TMA
// writes + operand reads) drops from 24 KiB to 16 KiB compared with the single-CTA 128 x 256 tile of gemm_tc.cu, and a
// stage takes 32 KiB instead of 48, which pays for a 6-deep ring (8 and 10 deep for 128 and 64 columns).  The leader CTA
// (cluster rank 0) issues every MMA; the accumulator rows [0, 128) live in the leader's TMEM and [128, 256) in the peer's,
// and each CTA's epilogue warps drain their own half.
//
//   warp 0 (both CTAs)  TMA producer: own halves of A and B (and the MXFP8 scale atoms) into own shared
//                       memory; the bytes of both CTAs are counted on the LEADER's "stage full" barrier
//   warp 1 (leader)     issues tcgen05.mma for the pair and commits to the leader's "stage empty" and "accumulator
//                       full" barriers; the leader's producer / first epilogue warp pass each of these on to the
//                       peer's barrier with a remote mbarrier arrive
//   warps 2..5 (both)   epilogue: TMEM -> registers -> bf16 -> shared memory -> whole lines in global memory; with an
//                       activation straight from the registers, in 32-byte sectors; every warp arrives on the
//                       leader's "accumulator empty" barrier (8 arrivals per tile)
//
// Warps 0 and 1 run their loops uniformly, with all lanes waiting; one elected lane issues.
//
// Every wait is bounded; on expiry the CTA raises its abort flag, all roles leave their loops, both CTAs meet
// at the closing cluster barrier (so neither exits while the other may still signal into it), TMEM is
// released and a device-side error word is set for the host, the communicator's status record too where the launch
// has one (the fused modes and the product of a one-rank plan).  No load is replicated across the cluster.
//
// Modes (as in gemm_tc.cu): the plain GEMM; all-gather -> GEMM, where extra CTAs of the grid move the peers' rows
// into local memory and each producer waits for the arrival counter of its own 128 rows; GEMM -> reduce-scatter,
// where the epilogue stores partial tiles into the row owner's staging area over NVLink and extra CTAs (then
// all CTAs) reduce this rank's rows.  The comm and reducer CTAs are the ones of gemm_tc.cu
// (gemm_fused_parts.cuh); they come in whole clusters and never take part in a cluster barrier.
//
// Operands may be stored transposed (bf16; a.ta, a.tb): the backward products of a linear layer contract over the
// dimension that is not contiguous.  TMA then fetches 64 x 64 boxes of [K, columns] and the MMA descriptors say
// MN-major, so nothing is copied first.  Making K-major copies of the six operands of an MLP's backward pass took
// 585 of the 1400 us of a training step (8192 x 4096 x 1792); the transposed forms run at the speed of the plain one.
//
// The reference has no compute kernels (README.md:5 only asks that collectives fuse with others).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../device/prims.cuh"
#include "../device/tc_prims.cuh"
#include "fused_schedule.h"
#include "gemm_fused_parts.cuh"
#include "gemm_tc.h"
#include "launch.h"

namespace mt {
using namespace tc;
namespace pair {

constexpr int BMC = 128;   // A rows (and accumulator rows) per CTA
constexpr int BM2 = 256;   // rows of the pair's tile
constexpr int kThreads = 192;
constexpr uint32_t A_BYTES = BMC * 128;   // rows of 128 bytes (64 bf16 or 128 fp8)
constexpr int EPI_PITCH = 144;
constexpr uint32_t EPI_BYTES = 4 * 32 * EPI_PITCH;
constexpr uint32_t CTL_BYTES = 512;
constexpr uint32_t TMEM_COLS = 512;
constexpr uint32_t T_CHUNK = 64 * 128;    // 64 K rows of 64 columns of an operand stored transposed

// Shared memory of one kernel form.  Narrow tiles move fewer bytes per k-block, so more stages keep as many in flight.
template <int MODE, bool FP8, int TILE_N, bool TB>
struct Shape {
  static constexpr int BNC = TILE_N / 2;   // B rows staged by each CTA
  static constexpr int STAGES = TILE_N >= 224 ? 6 : (TILE_N == 128 ? 8 : 10);
  static constexpr uint32_t B_BYTES = BNC * 128;   // a multiple of 1024: whole 128-byte swizzle atoms
  // transposed: whole 64-column chunks
  static constexpr uint32_t B_PITCH = TB ? (uint32_t)((BNC + 63) / 64) * T_CHUNK : B_BYTES;
  // MXFP8: scale atom of the CTA's A rows + those of all B rows of the tile
  static constexpr uint32_t SF_STAGE_BYTES = FP8 ? 512 * (1 + TILE_N / 128) : 0;
  static constexpr uint32_t RING = MODE == MODE_AG_GEMM ? fused::COMM_SLOTS * fused::COMM_PIECE : 0;   // comm CTAs reuse the stages
  static constexpr uint32_t OPERANDS = STAGES * (A_BYTES + B_PITCH) > RING ? STAGES * (A_BYTES + B_PITCH) : RING;
  static constexpr uint32_t SMEM = 1024 + OPERANDS + EPI_BYTES + CTL_BYTES + STAGES * SF_STAGE_BYTES;
  static_assert(SMEM <= 232448, "shared memory of one CTA");
};
constexpr int MAX_STAGES = 10;

struct Ctl {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full[2], acc_empty[2], drain;
  uint32_t tmem_base;
  int abort;
};
static_assert(sizeof(Ctl) <= CTL_BYTES && sizeof(fused::CommCtl) <= CTL_BYTES, "control block");
static_assert(kThreads == fused::kGemmThreads, "comm and reducer code assumes this block size");

__device__ int g_pair_error;  // set when a wait of this kernel expired (read by mt_gemm_pair_error)

__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint64_t timeout_ns) {
  uint32_t spins = 0;
  uint64_t t0 = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++spins & 0x3ffu) == 0) {
      if (*abort_flag) return false;
      const uint64_t now = globaltimer();
      if (t0 == 0) t0 = now;
      else if (now - t0 > timeout_ns) {
        *abort_flag = 1;
        return false;
      }
    }
  }
  return true;
}

// 32 bf16 of one row (64 bytes) in two 32-byte accesses, or in four of 16 bytes where the matrix is only aligned to that.
__device__ __forceinline__ void store_row64(uint8_t* p, const uint32_t* v, bool wide) {
  if (wide) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
      asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p + j * 32), "r"(v[8 * j]), "r"(v[8 * j + 1]),
                   "r"(v[8 * j + 2]), "r"(v[8 * j + 3]), "r"(v[8 * j + 4]), "r"(v[8 * j + 5]), "r"(v[8 * j + 6]), "r"(v[8 * j + 7])
                   : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) *(uint4*)(p + j * 16) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  }
}
__device__ __forceinline__ void load_row64(const uint8_t* p, uint32_t* v, bool wide) {
  if (wide) {
#pragma unroll
    for (int j = 0; j < 2; ++j)
      asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(v[8 * j]), "=r"(v[8 * j + 1]), "=r"(v[8 * j + 2]), "=r"(v[8 * j + 3]), "=r"(v[8 * j + 4]),
                     "=r"(v[8 * j + 5]), "=r"(v[8 * j + 6]), "=r"(v[8 * j + 7])
                   : "l"(p + j * 32));
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 t = *(const uint4*)(p + j * 16);
      v[4 * j] = t.x;
      v[4 * j + 1] = t.y;
      v[4 * j + 2] = t.z;
      v[4 * j + 3] = t.w;
    }
  }
}

// The same for a whole warp: one answer for all lanes, so that the issue loops stay warp-uniform.
__device__ __noinline__ bool wait_bar_warp_slow(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint64_t timeout_ns) {
  uint32_t spins = 0;
  uint64_t t0 = 0;
  while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
    if ((++spins & 0x3ffu) == 0) {
      if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
      const uint64_t now = __shfl_sync(0xffffffffu, globaltimer(), 0);
      if (t0 == 0) t0 = now;
      else if (now - t0 > timeout_ns) {
        *abort_flag = 1;
        return false;
      }
    }
  }
  return true;
}
__device__ __forceinline__ bool wait_bar_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint64_t timeout_ns) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return wait_bar_warp_slow(bar, parity, abort_flag, timeout_ns);
}
__device__ __forceinline__ bool aborted_warp(volatile int* abort_flag) { return __any_sync(0xffffffffu, *abort_flag != 0); }

// silu and its derivative on packed bf16: the bits that x / (1 + exp(-x)) and sig * (1 + x * (1 - sig)) have as separate fp32
// operations.  The quotients are Newton's iteration with Markstein's last correction (Computation of elementary functions on
// the IBM RISC System/6000 processor, 1990) on y / 4, which keeps 4 / y a normal number up to the largest y: no branches, so
// that the 32 elements of a step overlap.  CUDA's own quotient has a slow path for large y, which a lane in six takes where
// h is spread over +- 64: silu in the epilogue of 8192 x 1792 x 4096 then took 205 us, 88.8 this way
// (plain 83.0).  The fast exponential and quotient (87.3) are off by up to 1e-5 far from zero and flush silu to zero below
// -87.3, where bf16 still has values.
__device__ __forceinline__ float four_over(float y4) {   // 1 / y4 = 4 / y, y4 in [1 / 4, 2^126)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y4));
  return __fmaf_rn(r, __fmaf_rn(-y4, r, 1.f), r);
}
__device__ __forceinline__ float silu1(float x) {
  const float y = 1.f + expf(-x), y4 = 0.25f * y, x4 = 0.25f * x, r = four_over(y4), q0 = __fmul_rn(x4, r);
  const float q = fabsf(q0) <= 3.4028234e38f ? __fmaf_rn(__fmaf_rn(-y4, q0, x4), r, q0) : q0;   // x infinite or NaN: as it is
  return y <= 3.4028234e38f ? q : (y != y ? y : x * 0.f);                                       // y infinite: a zero
}
__device__ __forceinline__ float dsilu1(float d, float x) {
  const float y = 1.f + expf(-x);
  const float s = y <= 3.4028234e38f ? 0.25f * four_over(0.25f * y) : (y != y ? y : 0.f);
  return __fmul_rn(d, __fmul_rn(s, __fadd_rn(1.f, __fmul_rn(x, 1.f - s))));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *(uint32_t*)&p;
}
// 64 accumulator columns of this lane's row as packed bf16.
__device__ __forceinline__ void tmem_ld_pack64(uint32_t taddr, uint32_t* v) {
  uint32_t r0[32], r1[32];
  tmem_ld_32x32(taddr, r0);
  tmem_ld_32x32(taddr + 32, r1);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    v[j] = pack_bf16(__uint_as_float(r0[2 * j]), __uint_as_float(r0[2 * j + 1]));
    v[16 + j] = pack_bf16(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1]));
  }
}
__device__ __forceinline__ uint32_t silu2(uint32_t v) {
  return pack_bf16(silu1(__uint_as_float(v << 16)), silu1(__uint_as_float(v & 0xffff0000u)));
}
__device__ __forceinline__ uint32_t dsilu2(uint32_t d, uint32_t h) {
  return pack_bf16(dsilu1(__uint_as_float(d << 16), __uint_as_float(h << 16)),
                   dsilu1(__uint_as_float(d & 0xffff0000u), __uint_as_float(h & 0xffff0000u)));
}

// Tile order: fused_schedule.h with 256-row tiles (mb, jb count 256-row blocks).
using Tile = MtTile;
template <int MODE, int TILE_N>
__device__ __forceinline__ Tile tile_of(const GemmArgs& a, int lr, int t) {
  static_assert(MODE_PLAIN == MT_TILE_PLAIN && MODE_AG_GEMM == MT_TILE_AG_GEMM && MODE_GEMM_RS == MT_TILE_GEMM_RS, "mode codes");
  // a last block of 128 rows (plain GEMM) counts as a whole one: its peer CTA loads zeros and stores nothing
  return mt_fused_tile(MODE, t, MODE == MODE_PLAIN ? (a.M + BM2 - 1) & ~(BM2 - 1) : a.M, a.N, a.nranks, a.rank[lr], a.raster, BM2, TILE_N);
}

// TILE_N: columns of a tile.  256 moves the fewest operand bytes per product.  224 exists for the wave count: 8192 x 1792
// (the Llama-3-8B up projection on 8 ranks) is 224 tiles of 256 x 256, 3.03 waves on 74 clusters, i.e. a fourth wave for
// two tiles; as 256 tiles of 256 x 224 it is four waves of tiles that are an eighth smaller.  bf16 only (the MXFP8 scale
// atoms cover 128 rows of B) and not for GEMM -> reduce-scatter (its staging layout is in 256-column tiles).  128 and 64
// are for plain GEMMs that have too few 256-column tiles for the chip: a k-block of a narrow tile takes 0.55 / 0.4 of a
// wide one's time and two or four times as many SMs work (host rule: pick_plain_bn).
// A plain GEMM has one set of descriptors: 0.6 KB of kernel parameters instead of 5 (1 us of a launch).
template <int MODE>
constexpr int kMaps = MODE == MODE_PLAIN ? 1 : MT_MAX_RANKS;

// TA, TB: the operand is stored transposed (compile-time: choosing descriptors in the issue loops cost 7 %).
// EPI (GemmEpi): compile-time too, the code of the activations alone cost a plain 2048 x 4096 x 256 0.9 of 10.7 us.
template <int MODE, bool FP8, int TILE_N, bool TA = false, bool TB = false, int EPI = EPI_NONE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    gemm_pair_kernel(const __grid_constant__ GemmMapsN<kMaps<MODE>> maps, const __grid_constant__ PairSfMapsN<kMaps<MODE>> sfmaps,
                     GemmArgs a) {
  static_assert(TILE_N == 256 || (TILE_N == 224 && !FP8 && MODE != MODE_GEMM_RS) || (TILE_N == 128 && MODE == MODE_PLAIN) ||
                    (TILE_N == 64 && MODE == MODE_PLAIN && !FP8 && !TB), "tile widths");
  using S = Shape<MODE, FP8, TILE_N, TB>;
  constexpr int BN = TILE_N, BNC = S::BNC, STAGES = S::STAGES;
  constexpr uint32_t B_BYTES = S::B_BYTES, B_PITCH = S::B_PITCH, SF_STAGE_BYTES = S::SF_STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  const int lr = blockIdx.y;
  // through a shuffle: known to be the same in all lanes of the warp
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // the same offsets in both CTAs: the MMA descriptors name shared memory of the pair by offset
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * A_BYTES;
  uint8_t* sEpi = smem + S::OPERANDS;
  Ctl* ctl = (Ctl*)(sEpi + EPI_BYTES);
  uint8_t* sSF = sEpi + EPI_BYTES + CTL_BYTES;
  constexpr int BKE = FP8 ? 128 : 64;    // K elements per stage
  constexpr uint32_t ACC = FP8 && BN > 128 ? 1 : 2;  // accumulator buffers (MXFP8 keeps TMEM columns for the scales)
  const uint32_t cr = cluster_ctarank();
  const bool leader = cr == 0;
  const int nextra = MODE == MODE_PLAIN ? 0 : a.ncomm;  // AG: data movers, RS: dedicated reducers (whole clusters)
  const int ngemm = (int)gridDim.x - nextra;
  const int cluster_id = blockIdx.x >> 1, nclusters = ngemm >> 1;
  const uint64_t timeout_ns = a.timeout_ns;

  if (MODE == MODE_AG_GEMM && (int)blockIdx.x >= ngemm) {
    fused::ag_comm_cta<FP8>(a, lr, (int)blockIdx.x - ngemm, nextra, smem, (fused::CommCtl*)(sEpi + EPI_BYTES));
    return;
  }
  if (MODE == MODE_GEMM_RS && (int)blockIdx.x >= ngemm) {
    fused::rs_reduce_loop(a, lr);
    return;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&ctl->full[s], 1);   // the leader's producer arrives once with the byte count of both CTAs
      mbar_init(&ctl->empty[s], 1);  // leader: commit of the MMA thread; peer: arrive forwarded by the leader
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&ctl->acc_full[s], 1);
      mbar_init(&ctl->acc_empty[s], 8);  // 4 epilogue warps of each CTA
    }
    mbar_init(&ctl->drain, 1);
    ctl->abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&maps.a[lr]);
    tma_prefetch_desc(&maps.b[lr]);
  }
  if (warp == 1) {
    tmem_alloc_pair(&ctl->tmem_base, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anybody signals across
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);
  volatile int* abort_flag = &ctl->abort;

  static_assert(!(TA || TB || EPI) || !FP8, "8-bit operands are K-major and have no activation");
  const int tiles = ((a.M + BM2 - 1) / BM2) * (a.N / BN);
  const int kblocks = a.K / BKE;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs): a uniform warp, one lane issues
    {
      const uint32_t empty_peer = map_to_cta(smem_u32(&ctl->empty[0]), 1), full_leader = map_to_cta(smem_u32(&ctl->full[0]), 0);
      uint32_t s = 0, ph = 0;   // stage and its parity: running counters, no division in the issue loops
      bool passed = false;      // the ring has been round once
      for (int t = cluster_id; t < tiles && !aborted_warp(abort_flag); t += nclusters) {
        const Tile tc_ = tile_of<MODE, BN>(a, lr, t);
        int arow = tc_.mb * BM2 + (int)cr * BMC;
        const int brow = tc_.nb * BN + (int)cr * BNC;
        const int sfa_row = tc_.mb * 2 + (int)cr;  // 128-row block of A in the (gathered) scale tensor
        const CUtensorMap* amap = &maps.a[lr];
        if (MODE == MODE_AG_GEMM) {
          if (tc_.owner == a.rank[lr]) {
            amap = &maps.a2[lr];  // own rows come straight from the local shard
            arow -= tc_.owner * (a.M / a.nranks);
          } else {
            // this CTA's 128 rows were pushed by `owner`: wait until its comm CTAs have counted the block in
            const int per = (a.M / a.nranks) / BMC;
            const uint64_t* cnt = (const uint64_t*)a.flags_local[lr] + (uint64_t)tc_.owner * per + (tc_.jb * 2 + (int)cr);
            const uint64_t want = a.epoch * (uint64_t)a.comm_split;
            uint32_t spins = 0;
            uint64_t t0 = 0;
            while (load64_acquire_sys(cnt) < want) {   // every lane: each then orders its own loads behind the count
              if ((++spins & 0xffu) == 0) {
                const uint64_t now = globaltimer();
                if (t0 == 0) t0 = now;
                else if (now - t0 > timeout_ns || *abort_flag) {
                  *abort_flag = 1;
                  fused::gemm_report(a, lr, MT_WHERE_GEMM_FLAG);
                  break;
                }
              }
            }
            if (aborted_warp(abort_flag)) break;
            fence_proxy_async_global();  // peer stores (generic proxy) before our TMA reads (async proxy)
          }
        }
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!wait_bar_warp(&ctl->empty[s], ph ^ 1, abort_flag, timeout_ns)) break;
          if (elect_one()) {
            // the MMA thread's commit lands on the leader's barrier only: pass it on to the peer's producer
            if (leader && passed) mbar_arrive_cluster(empty_peer + s * 8);
            const uint32_t full0 = full_leader + s * 8;
            if (leader) mbar_expect_tx(&ctl->full[s], 2 * (A_BYTES + (TB ? B_PITCH : B_BYTES) + (FP8 ? SF_STAGE_BYTES : 0)));
            if (TA) {
              tma_load_2d_pair(sA + s * A_BYTES, amap, arow, kb * BKE, full0);
              tma_load_2d_pair(sA + s * A_BYTES + T_CHUNK, amap, arow + 64, kb * BKE, full0);
            } else {
              tma_load_2d_pair(sA + s * A_BYTES, amap, kb * BKE, arow, full0);
            }
            if (TB) {
              tma_load_2d_pair(sB + s * B_PITCH, &maps.b[lr], brow, kb * BKE, full0);
              if (BNC > 64) tma_load_2d_pair(sB + s * B_PITCH + T_CHUNK, &maps.b[lr], brow + 64, kb * BKE, full0);
            } else {
              tma_load_2d_pair(sB + s * B_PITCH, &maps.b[lr], kb * BKE, brow, full0);
            }
            if (FP8) {
              // scale atoms are rows of a [atoms, 128 x u32] tensor: atom (row block of 128, K block of 128)
              uint8_t* sf = sSF + s * SF_STAGE_BYTES;
              tma_load_2d_pair(sf, &sfmaps.sfa[lr], 0, sfa_row * kblocks + kb, full0);
              tma_load_2d_pair(sf + 512, &sfmaps.sfb[lr], 0, (tc_.nb * (BN / 128)) * kblocks + kb, full0);
              if (BN > 128) tma_load_2d_pair(sf + 1024, &sfmaps.sfb[lr], 0, (tc_.nb * 2 + 1) * kblocks + kb, full0);
            }
          }
          if (++s == STAGES) {
            s = 0;
            ph ^= 1;
            passed = true;
          }
        }
      }
      if (aborted_warp(abort_flag)) {
        // copies this warp issued may still be landing in shared memory: give them a bounded time
        const uint64_t t0 = globaltimer();
        while (globaltimer() - t0 < 100000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader): a uniform warp, one lane issues
    // What bounds a k-block of any width is this loop: with a single-lane branch around it every operand went through a
    // per-thread register, and wait, four MMAs and commit took 535 cycles (MXFP8, with its scale copies, 840) where the
    // tensor cores need 512 for a 256-column tile and a quarter of that for a 64-column one.
    if (leader) {
      constexpr uint32_t idesc = make_idesc_bf16(BM2, BN) | (TA ? kIdescTransA : 0u) | (TB ? kIdescTransB : 0u);
      constexpr uint32_t ka = TA ? 128 : 2, kb16 = TB ? 128 : 2;   // descriptor step of 16 elements along K
      const uint64_t da0 = TA ? make_smem_desc_mn_sw128(sA, T_CHUNK) : make_smem_desc_sw128(sA);
      const uint64_t db0 = TB ? make_smem_desc_mn_sw128(sB, T_CHUNK) : make_smem_desc_sw128(sB);
      const uint64_t dsf0 = make_smem_desc_sf(sSF);
      const uint32_t empty0 = smem_u32(&ctl->empty[0]);
      uint32_t s = 0, ph = 0, tile_i = 0;
      for (int t = cluster_id; t < tiles && !aborted_warp(abort_flag); t += nclusters, ++tile_i) {
        const uint32_t as = tile_i % ACC, aph = (tile_i / ACC) & 1;
        if (!wait_bar_warp(&ctl->acc_empty[as], aph ^ 1, abort_flag, timeout_ns)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + as * BN;
        bool ok = true;
        for (int kb = 0; kb < kblocks; ++kb) {
          if (!wait_bar_warp(&ctl->full[s], ph, abort_flag, timeout_ns)) {
            ok = false;
            break;
          }
          tc_fence_after();
          // descriptor addresses are in units of 16 bytes and stay below 2^14: no carry into the other fields
          const uint64_t da = da0 + s * (A_BYTES >> 4), db = db0 + s * (B_PITCH >> 4), dsf = dsf0 + s * (SF_STAGE_BYTES >> 4);
          const uint32_t tsfa = tmem_base + 256 + s * 16, tsfb = tsfa + 4, acc0 = kb > 0 ? 1u : 0u, bar = empty0 + s * 8;
          if (elect_one()) {
            if (FP8) {
              tmem_cp_sf_pair(tsfa, dsf);
              tmem_cp_sf_pair(tsfb, dsf + 32);
              if (BN > 128) tmem_cp_sf_pair(tsfb + 4, dsf + 64);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_mxfp8_pair(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), make_idesc_mxfp8(BM2, BN, k, k), tsfa,
                                tsfb, k > 0 ? 1u : acc0);
            } else {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                umma_bf16_pair(d_tmem, da + (uint64_t)(k * ka), db + (uint64_t)(k * kb16), idesc, k > 0 ? 1u : acc0);
            }
            // the stage is free (in both CTAs) once these MMAs have read it
            umma_commit_pair(bar);
          }
          if (++s == STAGES) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) break;
        if (elect_one()) umma_commit_pair(smem_u32(&ctl->acc_full[as]));
      }
      // no MMA may still be running when TMEM is freed, on the normal path or after an abort
      if (elect_one()) umma_commit_pair(smem_u32(&ctl->drain));
      wait_bar_warp(&ctl->drain, 0, abort_flag, timeout_ns);
    }
  } else {
    // ------------------------------------------------------------ epilogue warps (2..5, both CTAs)
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    uint8_t* stg = sEpi + (warp - 2) * 32 * EPI_PITCH;
    uint32_t tile_i = 0;
    for (int t = cluster_id; t < tiles; t += nclusters, ++tile_i) {
      const uint32_t as = tile_i % ACC, aph = (tile_i / ACC) & 1;
      if (!wait_bar(&ctl->acc_full[as], aph, abort_flag, timeout_ns)) break;
      // the commit lands on the leader's barrier only: its first epilogue warp passes it on to the peer
      if (leader && warp == 2 && lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&ctl->acc_full[as]), 1));
      tc_fence_after();
      const Tile tc_ = tile_of<MODE, BN>(a, lr, t);
      // destination of this CTA's 128 rows of the tile
      uint8_t* dst;
      uint64_t ld_bytes;
      uint64_t* rs_cnt = nullptr;
      if (MODE == MODE_GEMM_RS) {
        // partial tile -> staging[my rank] of the owner (peer memory unless the owner is this rank), tile-major:
        // [source rank][128-row block][column block][128 x 256], one contiguous 64 KiB region per CTA and tile
        const MtDevComm& c = a.comms[lr];
        const int per = (a.M / a.nranks) / BMC;
        const uint64_t slot = ((uint64_t)a.rank[lr] * per + (tc_.jb * 2 + (int)cr)) * (a.N / BN) + tc_.nb;
        ld_bytes = (uint64_t)BN * 2;
        dst = c.heap[tc_.owner] + a.stage_off + slot * (uint64_t)(BMC * BN * 2);
        rs_cnt = (uint64_t*)(c.heap[tc_.owner] + a.flags_off) + slot;
      } else {
        ld_bytes = (uint64_t)a.ldc * 2;
        dst = (uint8_t*)a.c[lr] + (uint64_t)(tc_.mb * BM2 + (int)cr * BMC) * ld_bytes + (uint64_t)tc_.nb * BN * 2;
      }
      dst += (uint64_t)(q * 32) * ld_bytes;
      const bool rows_out = MODE != MODE_PLAIN || tc_.mb * BM2 + (int)cr * BMC < a.M;   // M % 256 == 128: last peer has none
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + as * BN;
      const uint32_t acc_empty0 = map_to_cta(smem_u32(&ctl->acc_empty[as]), 0);
      // Whole 128-byte lines per store: 64 columns of the warp's 32 rows go through shared memory and leave as 4 rows per
      // pass of 8 lanes x 16 bytes (GEMM -> reduce-scatter: full NVLink packets).  Bound by the stores where K is small:
      // 32-byte sectors straight from each lane's row took 68.4 us for an MXFP8 8192 x 14336 x 256, lines take 56.2, and
      // 8192 x 4096 x 256 26.8 and 24.3 in bf16; from K = 1024 on, where the next tile's main loop hides the epilogue, both
      // are within 2 %.  `n16`: 16-byte pieces per row (4: the last 32 of 224 columns).
      // All 8 passes at once where the registers allow it (the fused MXFP8 kernels would spill; 4 cost the plain one 6 %).
      auto lines_out = [&](int cb, const uint32_t* v, int n16) {
        uint4* row = (uint4*)(stg + lane * EPI_PITCH);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < n16) row[j] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        __syncwarp();
#pragma unroll(FP8 && MODE != MODE_PLAIN ? 4 : 8)
        for (int p = 0; p < 8; ++p) {
          const int rr = p * 4 + (lane >> 3), c16 = lane & 7;
          if (c16 >= n16 || !rows_out) continue;
          const uint4 x = *(const uint4*)(stg + rr * EPI_PITCH + c16 * 16);
          uint8_t* g = dst + (uint64_t)rr * ld_bytes + cb * 128 + c16 * 16;
          if (MODE == MODE_GEMM_RS) {
            u128 w;
            w.x = (uint64_t)x.x | ((uint64_t)x.y << 32);
            w.y = (uint64_t)x.z | ((uint64_t)x.w << 32);
            store128_relaxed_sys(g, w);
          } else {
            *(uint4*)g = x;
          }
        }
        __syncwarp();
      };
      // accumulator drained: hand it back to the leader's MMA thread
      auto release_acc = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(acc_empty0);
      };
      if constexpr (FP8) {
        // drain the accumulator (256 columns: the only one) into registers (packed bf16) and hand it back, then store
        uint32_t pk[BN / 2];
#pragma unroll
        for (int cb = 0; cb < BN / 64; ++cb) tmem_ld_pack64(taddr + cb * 64, pk + cb * 32);
        release_acc();
#pragma unroll
        for (int cb = 0; cb < BN / 64; ++cb) lines_out(cb, pk + cb * 32, 8);
      } else if constexpr (EPI == EPI_NONE) {
#pragma unroll 1
        for (int cb = 0; cb < BN / 64; ++cb) {
          uint32_t pk[32];
          tmem_ld_pack64(taddr + cb * 64, pk);
          lines_out(cb, pk, 8);
        }
        if (BN % 64) {
          uint32_t r[32], pk[16];
          tmem_ld_32x32(taddr + BN / 64 * 64, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) pk[j] = pack_bf16(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
          lines_out(BN / 64, pk, 4);
        }
        release_acc();
      } else {
        // activation fused into the epilogue (the work overlaps the next tile's main loop): aux has C's layout, and every
        // lane keeps the row it got from TMEM and loads and stores it in whole 32-byte sectors
        const bool wide = a.wide_out != 0;
        uint8_t* row = dst + (uint64_t)lane * ld_bytes;
        uint8_t* aux = (uint8_t*)a.aux[lr] + (row - (uint8_t*)a.c[lr]);
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t r[32], v[16], h[16];
          if (EPI == EPI_DSILU && rows_out) load_row64(aux + c * 64, h, wide);
          tmem_ld_32x32(taddr + c * 32, r);
          tmem_ld_wait();
          if (c == BN / 32 - 1) release_acc();
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = pack_bf16(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
          if (!rows_out) continue;
          if (EPI == EPI_DSILU) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = dsilu2(v[j], h[j]);
          }
          store_row64(row + c * 64, v, wide);
          if (EPI == EPI_SILU) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = silu2(v[j]);
            store_row64(aux + c * 64, v, wide);
          }
        }
      }
      if (MODE == MODE_GEMM_RS) {
        // count this warp's quarter of the partial tile on the owner (release: the stores above come first)
        __syncwarp();
        if (lane == 0) asm volatile("red.release.sys.global.add.u64 [%0], %1;" ::"l"(rs_cnt), "l"(1ull) : "memory");
      }
    }
  }

  // ---------------------------------------------------------------- tear-down
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag) {
    // tell the peer (it would notice by itself after its own time limit) and the host
    st_cluster_u32(map_to_cta(smem_u32(&ctl->abort), cr ^ 1), 1u);
    atomicExch(&g_pair_error, 1);
    fused::gemm_report(a, lr, MT_WHERE_GEMM_FLAG);   // the plain GEMM has no status record, a one-rank plan does
  }
  cluster_sync_all();  // neither CTA leaves, or frees TMEM, while the other may still signal into it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
  // ---------------------------------------------------------------- reducer phase of GEMM -> reduce-scatter
  if (MODE == MODE_GEMM_RS) {
    if (*abort_flag) return;
    fused::rs_reduce_loop(a, lr);
  }
}

}  // namespace pair

// Forms of the bf16 kernels: operands as stored, and what the epilogue does.
enum PairForm { FORM_NN = 0, FORM_TB, FORM_TA_TB, FORM_SILU, FORM_TB_DSILU, FORM_COUNT };
struct PairKernel {
  const void* fn;
  uint32_t smem;
};
template <int MODE, bool FP8, int TILE_N, bool TA = false, bool TB = false, int EPI = EPI_NONE>
static PairKernel pair_kernel() {
  return {(const void*)pair::gemm_pair_kernel<MODE, FP8, TILE_N, TA, TB, EPI>, pair::Shape<MODE, FP8, TILE_N, TB>::SMEM};
}
template <bool TA, bool TB, int EPI>
static PairKernel plain_kernel(int bn) {
  switch (bn) {
    case 256: return pair_kernel<MODE_PLAIN, false, 256, TA, TB, EPI>();
    case 224: return pair_kernel<MODE_PLAIN, false, 224, TA, TB, EPI>();
    case 128: return pair_kernel<MODE_PLAIN, false, 128, TA, TB, EPI>();
    case 64:
      if constexpr (!TB) return pair_kernel<MODE_PLAIN, false, 64, TA, TB, EPI>();
      return {nullptr, 0};
    default: return {nullptr, 0};
  }
}
static PairKernel pair_fn(int mode, bool fp8, int bn = 256, int form = FORM_NN) {
  const PairKernel none = {nullptr, 0};
  if (fp8) {
    if (form != FORM_NN) return none;
    if (bn == 128) return mode == MODE_PLAIN ? pair_kernel<MODE_PLAIN, true, 128>() : none;
    if (bn != 256) return none;
    switch (mode) {
      case MODE_PLAIN: return pair_kernel<MODE_PLAIN, true, 256>();
      case MODE_AG_GEMM: return pair_kernel<MODE_AG_GEMM, true, 256>();
      case MODE_GEMM_RS: return pair_kernel<MODE_GEMM_RS, true, 256>();
      default: return none;
    }
  }
  if (mode == MODE_PLAIN) {
    switch (form) {
      case FORM_NN: return plain_kernel<false, false, EPI_NONE>(bn);
      case FORM_TB: return plain_kernel<false, true, EPI_NONE>(bn);
      case FORM_TA_TB: return plain_kernel<true, true, EPI_NONE>(bn);
      case FORM_SILU: return plain_kernel<false, false, EPI_SILU>(bn);
      case FORM_TB_DSILU: return plain_kernel<false, true, EPI_DSILU>(bn);
      default: return none;
    }
  }
  if (mode == MODE_AG_GEMM && (bn == 256 || bn == 224)) {
    const bool wide = bn == 256;
    if (form == FORM_NN) return wide ? pair_kernel<MODE_AG_GEMM, false, 256>() : pair_kernel<MODE_AG_GEMM, false, 224>();
    if (form == FORM_SILU)
      return wide ? pair_kernel<MODE_AG_GEMM, false, 256, false, false, EPI_SILU>()
                  : pair_kernel<MODE_AG_GEMM, false, 224, false, false, EPI_SILU>();
    return none;
  }
  if (mode == MODE_GEMM_RS && bn == 256) {
    if (form == FORM_TB) return pair_kernel<MODE_GEMM_RS, false, 256, false, true>();
    return form == FORM_NN ? pair_kernel<MODE_GEMM_RS, false, 256>() : none;
  }
  return none;
}
// The form a launch asks for, -1 where there is no such kernel.
static int form_of(const GemmArgs& a) {
  if (a.ta) return a.tb && a.epi == EPI_NONE ? FORM_TA_TB : -1;
  if (a.tb) return a.epi == EPI_NONE ? FORM_TB : (a.epi == EPI_DSILU ? FORM_TB_DSILU : -1);
  return a.epi == EPI_NONE ? FORM_NN : (a.epi == EPI_SILU ? FORM_SILU : -1);
}

// Clusters of this kernel that the device can hold at once.  The kernel is persistent (cluster i takes tiles
// i, i + n, ...), so a grid with more clusters than fit would run its tail after the rest has finished.
int gemm_pair_max_clusters(int mode, bool fp8, int bn, int form) {
  static int cached[3 * 2 * 4 * FORM_COUNT] = {};
  const PairKernel k = pair_fn(mode, fp8, bn, form);
  if (!k.fn) return 0;
  const int width = bn == 256 ? 0 : (bn == 224 ? 1 : (bn == 128 ? 2 : 3));
  int& slot = cached[((mode * 2 + (fp8 ? 1 : 0)) * 4 + width) * FORM_COUNT + form];
  if (slot > 0) return slot;
  if (cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem) != cudaSuccess) return 0;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(sms & ~1);
  cfg.blockDim = dim3(pair::kThreads);
  cfg.dynamicSmemBytes = k.smem;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = 2;
  at.val.clusterDim.y = 1;
  at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k.fn, &cfg) != cudaSuccess || n <= 0) {
    cudaGetLastError();
    n = sms / 2;
  }
  if (const char* e = getenv("MINTCCL_DEBUG")) {
    if (strcmp(e, "info") == 0 || strcmp(e, "trace") == 0 || atoi(e) > 0)  // same levels as the Python side
      fprintf(stderr, "[mintccl] pair GEMM (mode %d, %s): %d clusters of 2 CTAs fit on %d SMs\n", mode, fp8 ? "mxfp8" : "bf16", n, sms);
  }
  slot = n;
  return n;
}

// Grid: 2 * nclusters GEMM CTAs followed by a.ncomm comm / reducer CTAs (even), times nlocal emulated ranks.
cudaError_t launch_gemm_pair(int mode, const GemmMaps& maps, const PairSfMaps& sf, const GemmArgs& a, int nclusters,
                             int nlocal, cudaStream_t s, bool fp8, int bn) {
  const int form = form_of(a);
  const PairKernel k = form < 0 ? PairKernel{nullptr, 0} : pair_fn(mode, fp8, bn, form);
  if (!k.fn) return cudaErrorInvalidValue;
  const int fit = gemm_pair_max_clusters(mode, fp8, bn, form);  // also sets the shared-memory attribute once
  if (fit <= 0) return cudaErrorInvalidValue;
  const int extra = mode == MODE_PLAIN ? 0 : a.ncomm;
  if (extra & 1) return cudaErrorInvalidValue;
  if ((nclusters + extra / 2) * nlocal > fit) nclusters = fit / nlocal - extra / 2;
  if (nclusters < 1) return cudaErrorInvalidValue;
  GemmMaps m;
  PairSfMaps sm;
  GemmMapsN<1> m1;
  PairSfMapsN<1> sm1;
  if (mode == MODE_PLAIN) {
    m1.a[0] = maps.a[0];
    m1.b[0] = maps.b[0];
    m1.a2[0] = maps.a2[0];
    sm1.sfa[0] = sf.sfa[0];
    sm1.sfb[0] = sf.sfb[0];
  } else {
    m = maps;
    sm = sf;
  }
  GemmArgs args = a;
  uint64_t mis = (uint64_t)a.ldc * 2;
  for (int lr = 0; lr < nlocal; ++lr) mis |= (uint64_t)(uintptr_t)a.c[lr] | (uint64_t)(uintptr_t)a.aux[lr];
  args.wide_out = (mis & 31) == 0;
  void* p[] = {mode == MODE_PLAIN ? (void*)&m1 : (void*)&m, mode == MODE_PLAIN ? (void*)&sm1 : (void*)&sm, (void*)&args};
  count_launch();
  const dim3 grid(2 * nclusters + extra, nlocal);
  if (nlocal == 1) return cudaLaunchKernel(k.fn, grid, dim3(pair::kThreads), p, k.smem, s);
  // emulated ranks wait on each other inside one grid: every CTA has to be resident
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = dim3(pair::kThreads);
  cfg.dynamicSmemBytes = k.smem;
  cfg.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeCooperative;
  at.val.cooperative = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, k.fn, p);
}

int gemm_pair_error() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, pair::g_pair_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // namespace mt
