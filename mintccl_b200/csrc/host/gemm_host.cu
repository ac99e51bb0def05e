// Host side of the tcgen05 GEMM kernels: TMA descriptors, argument checks, launches.
#include <cuda.h>
#include <cuda_runtime.h>
#include <limits.h>
#include <string.h>

#include <string>

#include "../kernels/gemm_tc.h"
#include "../kernels/mxfp8.h"
#include "comm_internal.h"

using mthost::fail;

namespace {

constexpr int kBM = 128, kBN = 256, kBK = 64;
constexpr int kPairDefault = 1;  // plain GEMMs on CTA pairs unless MINTCCL_GEMM_PAIR says otherwise

// The encoder wants a current context.  A thread whose first CUDA call this is has none yet (autograd's backward
// threads): bind its device and try again.
template <class F>
CUresult with_context(F encode) {
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT || r == CUDA_ERROR_NOT_INITIALIZED) {
    int dev = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
  }
  return r;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// [rows, K] bf16 row-major, tiles of box_rows x 64 elements, 128-byte swizzle.
int make_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint32_t box_rows, bool fp8 = false) {
  static EncodeTiledFn enc = (EncodeTiledFn)mthost::driver_entry("cuTensorMapEncodeTiled");
  if (!enc) return fail("cuTensorMapEncodeTiled not available");
  const uint64_t esz = fp8 ? 1 : 2;
  if (((uintptr_t)base & 15) || (K * esz) % 16) return fail("GEMM operands must be 16-byte aligned with rows a multiple of 16 bytes");
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {K * esz};
  cuuint32_t box[2] = {(cuuint32_t)(fp8 ? 128 : kBK), box_rows};  // 128 bytes per row either way
  cuuint32_t estr[2] = {1, 1};
  CUresult r = with_context([&] { return enc(map, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE); });
  if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled failed: CUresult " + std::to_string((int)r));
  return 0;
}

// [K, cols] bf16 row-major (an operand stored transposed), boxes of 64 columns x 64 K rows, 128-byte swizzle.
int make_map_t(CUtensorMap* map, const void* base, uint64_t K, uint64_t cols) {
  static EncodeTiledFn enc = (EncodeTiledFn)mthost::driver_entry("cuTensorMapEncodeTiled");
  if (!enc) return fail("cuTensorMapEncodeTiled not available");
  if (((uintptr_t)base & 15) || (cols * 2) % 16) return fail("GEMM operands must be 16-byte aligned with rows a multiple of 16 bytes");
  cuuint64_t dims[2] = {cols, K};
  cuuint64_t strides[1] = {cols * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)kBK};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = with_context([&] { return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE); });
  if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled (transposed) failed: CUresult " + std::to_string((int)r));
  return 0;
}

// Tiled MXFP8 scales as a [atoms, 128] tensor of 32-bit words: one box = one 512-byte atom.
int make_sf_map(CUtensorMap* map, const void* base, uint64_t atoms) {
  static EncodeTiledFn enc = (EncodeTiledFn)mthost::driver_entry("cuTensorMapEncodeTiled");
  if (!enc) return fail("cuTensorMapEncodeTiled not available");
  if ((uintptr_t)base & 15) return fail("scale tensors must be 16-byte aligned");
  cuuint64_t dims[2] = {128, atoms};
  cuuint64_t strides[1] = {512};
  cuuint32_t box[2] = {128, 1};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = with_context([&] { return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE); });
  if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled (scales) failed: CUresult " + std::to_string((int)r));
  return 0;
}

int check_shape(int M, int N, int K, int nranks) {
  if (M <= 0 || N <= 0 || K <= 0) return fail("bad GEMM shape");
  if (M % (kBM * nranks) || N % kBN || K % kBK)
    return fail("GEMM shape: M must be a multiple of 128 x ranks, N of 256, K of 64");
  return 0;
}

int sm_count(int device) {
  int n = 148;
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device);
  return n;
}

}  // namespace

namespace mthost {
int make_bf16_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t K, uint32_t box_rows) {
  return make_map(map, base, rows, K, box_rows);
}
}  // namespace mthost

// Row blocks per group of the plain GEMM's tile order.  Row-major order streams the whole of B through the
// L2 once per wave of CTAs; when B does not fit beside A's rows (large N x K) a grouped order keeps a wave's
// operands resident.  MINTCCL_GEMM_RASTER overrides (for tuning).
static int raster_for(int /*M*/, int N, int K, int elem_bytes) {
  if (const char* e = getenv("MINTCCL_GEMM_RASTER")) return atoi(e);
  const double b_bytes = (double)N * K * elem_bytes;
  return b_bytes > 48e6 ? 16 : 1;
}

// GEMMs run on CTA pairs (gemm_tc2.cu); the fused kernels when a rank's rows are a multiple of 256, plain ones as gemm_plain
// says.  MINTCCL_GEMM_PAIR=0: the single-CTA kernels of gemm_tc.cu.
static int g_pair_mode = -1;
static bool pair_on() {
  if (g_pair_mode < 0) {
    const char* e = getenv("MINTCCL_GEMM_PAIR");
    g_pair_mode = e ? atoi(e) : kPairDefault;
  }
  return g_pair_mode != 0;
}
static bool use_pair(int M) { return pair_on() && M % 256 == 0; }

// Tile width of a bf16 pair GEMM over `row_tiles` 256-row blocks on `nclusters` clusters: 224 columns when N
// allows it and the waves of narrower tiles add up to less work than the waves of 256-column tiles.
static int pick_wide(int row_tiles, int N, int nclusters, bool fp8) {
  if (fp8 || N % 224 || nclusters < 1) return 256;
  const long w256 = (long)((row_tiles * (N / 256) + nclusters - 1) / nclusters) * 256;
  const long w224 = (long)((row_tiles * (N / 224) + nclusters - 1) / nclusters) * 224;
  return w224 < w256 ? 224 : 256;
}
// The environment's tile width (MINTCCL_GEMM_BN), where the kernel has it; 0: none.
static int forced_bn(int N, bool fp8, bool plain, bool tb) {
  const char* e = getenv("MINTCCL_GEMM_BN");
  const int v = e ? atoi(e) : 0;
  if (v == 256 || (v == 224 && !fp8 && N % 224 == 0) || (plain && v == 128) || (plain && v == 64 && !fp8 && !tb)) return v;
  return 0;
}
static int pick_bn(int row_tiles, int N, int nclusters, bool fp8) {
  const int f = forced_bn(N, fp8, false, false);
  return f ? f : pick_wide(row_tiles, N, nclusters, fp8);
}
// The same for a plain GEMM, where narrow tiles are to be had too.  The time of a wave in tenths of a 256-column k-block
// (580 cycles): 9 a k-block for 224 columns, 5.5 for 128 (290 - 320 cycles), 4 for 64 (220: A's bytes do not shrink with
// the tile), and one k-block to drain the last accumulator; an MXFP8 k-block of 128 elements has the same ratios.  So a
// problem with too few wide tiles for the chip takes the widest ones that fill it.  Of 204 shapes of whole 256-row blocks
// (256, 2048 and 8192 rows, 256 - 14336 columns, K = 256 - 8192, both types), timed in every width, the choice is within 5 %
// of the best for all but one (8192 x 14336 x 256: 9 %).  Measured (us, 256 / 128 / 64 columns): 256 x 4096 x 2048 16.6 /
// 12.5 / 10.4, 2048 x 1024 x 4096 27.1 / 18.6 / 23.3, 2048 x 4096 x 2048 28.9 / 28.8 / 37.1, 8192 x 1792 x 4096 90.1 / 87.6 /
// 117.4 (224: 84.6); MXFP8 (256 / 128) 256 x 1792 x 4096 16.6 / 11.3, 8192 x 1792 x 4096 51.3 / 48.5, 8192 x 4096 x 2048
// 53.8 / 57.1.
static int pick_plain_bn(int row_tiles, int N, int kblocks, int nclusters, bool fp8, bool tb, long* cost_out = nullptr) {
  if (const int f = forced_bn(N, fp8, true, tb)) return f;
  const int wide = pick_wide(row_tiles, N, nclusters, fp8);
  if (nclusters < 1) return wide;
  auto cost = [&](int bn, int per2) {   // twice the tenths
    return (long)((row_tiles * (N / bn) + nclusters - 1) / nclusters) * (kblocks * per2 + 20);
  };
  int best = wide;
  long c = cost(wide, wide == 224 ? 18 : 20);
  if (cost(128, 11) < c) {
    best = 128;
    c = cost(128, 11);
  }
  if (!fp8 && !tb && cost(64, 8) < c) {
    best = 64;
    c = cost(64, 8);
  }
  if (cost_out) *cost_out = c;
  return best;
}
// Clusters that `sms` SMs give a plain pair GEMM.
static int pair_clusters(int sms, bool fp8) {
  const int fit = mt::gemm_pair_max_clusters(mt::MODE_PLAIN, fp8), ncl = sms / 2;
  return fit > 0 && ncl > fit ? fit : ncl;
}

// How long a wait inside a product may take, and the status record that learns of one that took longer: those of the
// communicator whose one-rank plan it stands in for; by default 4 s and none (mt_gemm_pair_error).
struct Waits {
  uint64_t timeout_ns = 4000000000ull;
  void* status = nullptr;
  int rank = 0;
};
static Waits waits_of(const mt::GemmArgs& plan) { return {plan.timeout_ns, plan.status[0], plan.rank[0]}; }

static mt::GemmArgs product_args(void* C, int M, int N, int K, int ldc, const Waits& waits) {
  mt::GemmArgs a;
  memset(&a, 0, sizeof(a));
  a.c[0] = C;
  a.M = M;
  a.N = N;
  a.K = K;
  a.ldc = ldc;
  a.nranks = 1;
  a.timeout_ns = waits.timeout_ns;
  a.status[0] = waits.status;
  a.rank[0] = waits.rank;
  return a;
}

static int gemm_pair(void* stream, const void* A, const void* sfa, const void* B, const void* sfb, void* C, int M, int N,
                     int K, int ldc, int nctas, bool fp8, int stat, const Waits& waits, bool ta = false, bool tb = false,
                     int epi = mt::EPI_NONE, void* aux = nullptr) {
  int dev = 0;
  cudaGetDevice(&dev);
  const int row_tiles = (M + 255) / 256;
  const int ncl = pair_clusters(nctas > 0 ? nctas : sm_count(dev), fp8);
  const int bn = pick_plain_bn(row_tiles, N, K / (fp8 ? 128 : 64), ncl, fp8, tb);
  mt::GemmMaps maps;
  mt::PairSfMaps sf;
  memset(&maps, 0, sizeof(maps));
  memset(&sf, 0, sizeof(sf));
  if (ta ? make_map_t(&maps.a[0], A, K, M) : make_map(&maps.a[0], A, M, K, 128, fp8)) return -1;
  if (tb ? make_map_t(&maps.b[0], B, K, N) : make_map(&maps.b[0], B, N, K, bn / 2, fp8)) return -1;
  maps.a2[0] = maps.a[0];
  if (fp8) {
    if (make_sf_map(&sf.sfa[0], sfa, (uint64_t)(M / 128) * (K / 128)) ||
        make_sf_map(&sf.sfb[0], sfb, (uint64_t)(N / 128) * (K / 128)))
      return -1;
  }
  mt::GemmArgs a = product_args(C, M, N, K, ldc, waits);
  a.ta = ta;
  a.tb = tb;
  a.epi = epi;
  a.aux[0] = aux;
  a.raster = raster_for(M, N, K, fp8 ? 1 : 2) / 2;
  const int tiles = row_tiles * (N / bn);
  int nclusters = (nctas > 0 ? nctas : sm_count(dev)) / 2;
  if (nclusters > tiles) nclusters = tiles;
  if (nclusters < 1) nclusters = 1;
  cudaError_t e = mt::launch_gemm_pair(mt::MODE_PLAIN, maps, sf, a, nclusters, 1, (cudaStream_t)stream, fp8, bn);
  if (e != cudaSuccess) return fail(std::string("pair gemm launch: ") + cudaGetErrorString(e));
  mthost::stat_add(stat, (uint64_t)(2.0 * M * N * K));
  return 0;
}

// The same product on single CTAs (128 x 256 tiles), K-major operands.
static int gemm_single(void* stream, const void* A, const void* sfa, const void* B, const void* sfb, void* C, int M, int N, int K,
                       int ldc, int nctas, bool fp8, int stat, const Waits& waits) {
  int dev = 0;
  cudaGetDevice(&dev);
  mt::GemmMaps maps;
  memset(&maps, 0, sizeof(maps));
  if (make_map(&maps.a[0], A, M, K, kBM, fp8) || make_map(&maps.b[0], B, N, K, kBN, fp8)) return -1;
  maps.a2[0] = maps.a[0];
  mt::GemmArgs a = product_args(C, M, N, K, ldc, waits);
  a.sfa[0] = sfa;
  a.sfb[0] = sfb;
  a.raster = raster_for(M, N, K, fp8 ? 1 : 2);
  const int tiles = (M / kBM) * (N / kBN);
  int grid = nctas > 0 ? nctas : sm_count(dev);
  if (grid > tiles) grid = tiles;
  cudaError_t e = mt::launch_gemm_tc(mt::MODE_PLAIN, maps, a, grid, 1, (cudaStream_t)stream, fp8);
  if (e != cudaSuccess) return fail(std::string("gemm launch: ") + cudaGetErrorString(e));
  mthost::stat_add(stat, (uint64_t)(2.0 * M * N * K));
  return 0;
}

// C[M, ldc] = A[M, K] * B[N, K]^T, both K-major, on the kernel that suits the shape.  A last block of 128 rows leaves half a
// pair idle, and 128-row tiles of single CTAs can need a wave less (1152 x 4096: 144 tiles on 148 SMs; pairs have 80 on 74
// clusters).  In pick_plain_bn's unit (twice the tenths of a 256-column k-block) a wave of single CTAs costs 23 a k-block
// and 5 (10 in MXFP8) for the drain; a lone bf16 wave 20.7 and 24 less, since nothing waits for its accumulator.  Of 418
// shapes with 128 leftover rows (128 - 4224 x 256 - 14336, K = 256 - 8192, both types), timed on both kernels with operands
// in the L2, six lose 4 - 7 % by this choice and the others at most 3.  1152 x 4096 x 4096 takes 28.9 us (pairs 38.0), MXFP8
// 1152 x 4096 x 1024 10.4 (12.5); 2176 x 14336 x 1024 stays on pairs: 49.0, single CTAs 54.1.  A lone wave is left to pairs
// from K = 4096 on, where operands that come from HBM decide: 640 x 4096 x 4096 28.8 us on pairs and 30.8 on single CTAs
// (28.8 and 26.8 out of the L2), 4224 x 1024 x 4096 29.7 and 31.9.
static long single_cost(int M, int N, int kblocks, int sms, bool fp8) {
  const long waves = ((long)(M / kBM) * (N / kBN) + sms - 1) / sms;
  if (waves == 1 && !fp8) return kblocks * 207L / 10 - 24;
  return waves * (kblocks * 23L + (fp8 ? 10 : 5));
}
static int gemm_plain(void* stream, const void* A, const void* sfa, const void* B, const void* sfb, void* C, int M, int N, int K,
                      int ldc, int nctas, bool fp8, int stat, const Waits& waits = Waits()) {
  bool single = !pair_on();
  if (!single && M % 256 && !forced_bn(N, fp8, true, false)) {
    int dev = 0;
    cudaGetDevice(&dev);
    const int sms = nctas > 0 ? nctas : sm_count(dev), kblocks = K / (fp8 ? 128 : 64);
    long pairs = LONG_MAX;   // fewer than two CTAs asked for: no pair
    pick_plain_bn((M + 255) / 256, N, kblocks, pair_clusters(sms, fp8), fp8, false, &pairs);
    single = single_cost(M, N, kblocks, sms, fp8) < pairs;
  }
  return single ? gemm_single(stream, A, sfa, B, sfb, C, M, N, K, ldc, nctas, fp8, stat, waits)
                : gemm_pair(stream, A, sfa, B, sfb, C, M, N, K, ldc, nctas, fp8, stat, waits);
}

extern "C" {

// 1 after a bounded wait of the CTA-pair GEMM expired (the result of that call is then invalid), 0 otherwise.
int mt_gemm_pair_error(void) { return mt::gemm_pair_error(); }
// 1: plain GEMMs use CTA pairs where the shape allows, 0: single-CTA kernel, -1: back to the environment / default.
void mt_gemm_set_pair(int mode) { g_pair_mode = mode; }

// C[M, ldc] = A[M, K] * B[N, K]^T in bf16 with fp32 accumulation, on the current device.
int mt_gemm(void* stream, const void* A, const void* B, void* C, int M, int N, int K, int ldc, int nctas) {
  if (check_shape(M, N, K, 1)) return -1;
  if (ldc < N || ldc % 8 || ((uintptr_t)C & 15)) return fail("C must be 16-byte aligned with ldc >= N, ldc % 8 == 0");
  return gemm_plain(stream, A, nullptr, B, nullptr, C, M, N, K, ldc, nctas, false, mthost::ST_GEMM);
}

// C[M, N] = A * B in bf16 with fp32 accumulation, where either operand may be stored transposed: A as [K, M] (ta) or
// [M, K], B as [K, N] (tb) or [N, K].  Always on CTA pairs.
int mt_gemm_t(void* stream, const void* A, const void* B, void* C, int M, int N, int K, int ta, int tb) {
  if (check_shape(M, N, K, 1)) return -1;
  if ((uintptr_t)C & 15) return fail("C must be 16-byte aligned");
  return gemm_pair(stream, A, nullptr, B, nullptr, C, M, N, K, N, 0, false, mthost::ST_GEMM, Waits(), ta != 0, tb != 0);
}
// C[M, N] = (A[M, K] * B[K, N]) * silu'(H[M, N]): the gradient through silu and the layer behind it.
int mt_gemm_dsilu(void* stream, const void* A, const void* B, const void* H, void* C, int M, int N, int K) {
  if (check_shape(M, N, K, 1)) return -1;
  if (((uintptr_t)C | (uintptr_t)H) & 15) return fail("C and H must be 16-byte aligned");
  return gemm_pair(stream, A, nullptr, B, nullptr, C, M, N, K, N, 0, false, mthost::ST_GEMM, Waits(), false, true, mt::EPI_DSILU, (void*)H);
}
// Do problems of `rows` rows per rank run on CTA pairs (the kernels that take a transposed B)?
int mt_gemm_uses_pair(int rows) { return use_pair(rows) ? 1 : 0; }

// C[M, ldc] (bf16) = (A * SFA)[M, K] * (B * SFB)[N, K]^T for MXFP8 operands: e4m3 payload, ue8m0 scales per 32
// elements along K.  The scales are given in the tiled layout the tensor core reads: [rows / 128][K / 128][512]
// with byte (r % 32) * 16 + ((r % 128) / 32) * 4 + (k / 32) % 4 for row r and element k
// (mintccl_b200.ops.mxfp8.tile_scales builds it).  K must be a multiple of 128.
int mt_gemm_mxfp8(void* stream, const void* A, const void* sfa, const void* B, const void* sfb, void* C, int M, int N,
                  int K, int ldc, int nctas) {
  if (check_shape(M, N, K, 1) || K % 128) return fail("MXFP8 GEMM: M multiple of 128, N of 256, K of 128");
  if (ldc < N || ldc % 8 || ((uintptr_t)C & 15)) return fail("C must be 16-byte aligned with ldc >= N, ldc % 8 == 0");
  if (((uintptr_t)sfa | (uintptr_t)sfb) & 15) return fail("scale tensors must be 16-byte aligned");
  return gemm_plain(stream, A, sfa, B, sfb, C, M, N, K, ldc, nctas, true, mthost::ST_GEMM_MXFP8);
}

static int fused_common(MtComm* c, mt::GemmArgs& a, int M, int N, int K, uint64_t flags_off, uint64_t epoch) {
  if (!c || !c->d_comms) return fail("communicator is not finalized");
  if (check_shape(M, N, K, c->nranks)) return -1;
  memset(&a, 0, sizeof(a));
  a.M = M;
  a.N = N;
  a.K = K;
  a.nranks = c->nranks;
  a.comms = c->d_comms;
  a.flags_off = flags_off;
  a.epoch = epoch;
  a.timeout_ns = c->timeout_ns;
  for (int lr = 0; lr < c->nlocal; ++lr) {
    const int r = c->emulated ? lr : c->rank;
    a.rank[lr] = r;
    a.status[lr] = c->heap[lr][r] + c->L.status_off;
  }
  return 0;
}

// Host-side check of what a one-rank plan's product is launched with: out = {time limit, status record, rank}.
int mt_test_one_rank_args(uint64_t timeout_ns, void* heap, uint64_t status_off, uint64_t* out) {
  MtComm c;
  c.timeout_ns = timeout_ns;
  c.heap[0][0] = (uint8_t*)heap;
  c.L.status_off = status_off;
  c.d_comms = (MtDevComm*)heap;
  mt::GemmArgs plan;
  if (fused_common(&c, plan, 128, 256, 64, 0, 1)) return -1;
  const mt::GemmArgs a = product_args(nullptr, 128, 256, 64, 256, waits_of(plan));
  out[0] = a.timeout_ns;
  out[1] = (uint64_t)(uintptr_t)a.status[0];
  out[2] = (uint64_t)a.rank[0];
  return 0;
}

// C[M, ldc] = allgather(a_shard)[M, K] * B[N, K]^T.  `gather_off`: symmetric buffer of M * K bf16;
// `flags_off`: symmetric u64 counters [ranks][M / ranks / 128], zero before the first call; `epoch`: 1 on the
// first call on these counters, then 2, 3, ...; `ncomm` must not change between calls on the same counters.
static int ag_gemm_impl(MtComm* c, void* stream, const void* const* a_shard, const void* const* B, void* const* C,
                        uint64_t gather_off, uint64_t flags_off, uint64_t epoch, int M, int N, int K, int ldc, int ncomm,
                        int nctas, int comm_mode, uint64_t shard_off, int comm_split, bool fp8, const void* const* sfa,
                        const void* const* sfb, void* const* act = nullptr) {
  mt::GemmArgs a;
  if (fp8 && K % 128) return fail("MXFP8: K must be a multiple of 128");
  if (fused_common(c, a, M, N, K, flags_off, epoch)) return -1;
  if (ldc < N || ldc % 8) return fail("ldc must be >= N and a multiple of 8");
  const int n = c->nranks;
  if (act) {
    for (int lr = 0; lr < c->nlocal; ++lr) {
      if (((uintptr_t)C[lr] | (uintptr_t)act[lr]) & 15) return fail("C and the activation must be 16-byte aligned");
      a.aux[lr] = act[lr];
    }
    a.epi = mt::EPI_SILU;
    if (n > 1 && (!use_pair(M / n) || comm_mode == 2)) return fail("the fused activation runs on CTA pairs");
  }
  if (comm_mode < 0 || comm_mode > 3) return fail("comm_mode must be 0, 1, 2 or 3");
  if (n == 1) {   // nothing to gather: the product itself (gather_off, flags_off and epoch are not looked at)
    if (nctas == 1 && use_pair(M) && comm_mode != 2) return fail("not enough CTAs for the requested comm CTAs");
    if (((uintptr_t)C[0] & 15) || (fp8 && (((uintptr_t)sfa[0] | (uintptr_t)sfb[0]) & 15))) return fail("C and the scales must be 16-byte aligned");
    if (!act)
      return gemm_plain(stream, a_shard[0], fp8 ? sfa[0] : nullptr, B[0], fp8 ? sfb[0] : nullptr, C[0], M, N, K, ldc, nctas, fp8,
                        mthost::ST_AG_GEMM, waits_of(a));
    return gemm_pair(stream, a_shard[0], nullptr, B[0], nullptr, C[0], M, N, K, ldc, nctas, false, mthost::ST_AG_GEMM, waits_of(a),
                     false, false, a.epi, a.aux[0]);
  }
  if (ncomm < 1 || ncomm > 64) return fail("ncomm out of range");
  int grid = nctas > 0 ? nctas : sm_count(c->device);
  if (c->emulated && grid * c->nlocal > sm_count(c->device)) grid = sm_count(c->device) / c->nlocal;
  if (grid <= ncomm) return fail("not enough CTAs for the requested comm CTAs");
  if (ncomm > MT_MAX_BAR_SLOTS) return fail("too many comm CTAs");
  a.ldc = ldc;
  a.ncomm = ncomm;
  a.gather_off = gather_off;
  a.comm_mode = comm_mode;
  if (comm_split < 1 || comm_split > ncomm) return fail("comm_split must be in [1, ncomm]");
  a.comm_split = comm_split;
  a.shard_off = shard_off;
  mt::GemmMaps maps;
  memset(&maps, 0, sizeof(maps));
  for (int lr = 0; lr < c->nlocal; ++lr) {
    const int r = a.rank[lr];
    a.c[lr] = C[lr];
    a.a_local[lr] = a_shard[lr];
    a.flags_local[lr] = c->heap[lr][r] + flags_off;
    if (make_map(&maps.a[lr], c->heap[lr][r] + gather_off, M, K, kBM, fp8) || make_map(&maps.b[lr], B[lr], N, K, kBN, fp8) ||
        make_map(&maps.a2[lr], a_shard[lr], M / n, K, kBM, fp8))
      return -1;
    if ((uintptr_t)C[lr] & 15) return fail("C must be 16-byte aligned");
    if (fp8) {
      a.sfa[lr] = sfa[lr];
      a.sfb[lr] = sfb[lr];
    }
  }
  if (use_pair(M / n) && comm_mode != 2) {
    // CTA pairs: 256-row tiles inside one owner's rows, B split between the two CTAs, comm CTAs in whole clusters
    mt::PairSfMaps sf;
    memset(&sf, 0, sizeof(sf));
    a.ncomm = (ncomm + 1) & ~1;
    if (a.comm_split > 1 && a.ncomm % a.comm_split) return fail("comm_split must divide the (even) number of comm CTAs");
    const int nclusters = (grid - a.ncomm) / 2;
    if (nclusters < 1) return fail("not enough CTAs for the requested comm CTAs");
    const int bn = pick_bn(M / 256, N, nclusters, fp8);
    for (int lr = 0; lr < c->nlocal; ++lr) {
      if (make_map(&maps.b[lr], B[lr], N, K, bn / 2, fp8)) return -1;
      if (fp8 && (make_sf_map(&sf.sfa[lr], sfa[lr], (uint64_t)(M / 128) * (K / 128)) ||
                  make_sf_map(&sf.sfb[lr], sfb[lr], (uint64_t)(N / 128) * (K / 128))))
        return -1;
    }
    cudaError_t e2 = mt::launch_gemm_pair(mt::MODE_AG_GEMM, maps, sf, a, nclusters, c->nlocal, (cudaStream_t)stream, fp8, bn);
    if (e2 != cudaSuccess) return fail(std::string("pair ag_gemm launch: ") + cudaGetErrorString(e2));
    mthost::stat_add(mthost::ST_AG_GEMM, (uint64_t)(2.0 * M * N * K));
    return 0;
  }
  cudaError_t e = mt::launch_gemm_tc(mt::MODE_AG_GEMM, maps, a, grid, c->nlocal, (cudaStream_t)stream, fp8);
  if (e != cudaSuccess) return fail(std::string("ag_gemm launch: ") + cudaGetErrorString(e));
  mthost::stat_add(mthost::ST_AG_GEMM, (uint64_t)(2.0 * M * N * K));
  return 0;
}

int mt_ag_gemm(MtComm* c, void* stream, const void* const* a_shard, const void* const* B, void* const* C,
               uint64_t gather_off, uint64_t flags_off, uint64_t epoch, int M, int N, int K, int ldc, int ncomm,
               int nctas, int comm_mode, uint64_t shard_off, int comm_split) {
  return ag_gemm_impl(c, stream, a_shard, B, C, gather_off, flags_off, epoch, M, N, K, ldc, ncomm, nctas, comm_mode,
                      shard_off, comm_split, false, nullptr, nullptr);
}
// The same with act[M, ldc] = silu(C) from the epilogue (C as rounded to bf16).
int mt_ag_gemm_silu(MtComm* c, void* stream, const void* const* a_shard, const void* const* B, void* const* C, void* const* act,
                    uint64_t gather_off, uint64_t flags_off, uint64_t epoch, int M, int N, int K, int ldc, int ncomm,
                    int nctas, int comm_mode, uint64_t shard_off, int comm_split) {
  return ag_gemm_impl(c, stream, a_shard, B, C, gather_off, flags_off, epoch, M, N, K, ldc, ncomm, nctas, comm_mode,
                      shard_off, comm_split, false, nullptr, nullptr, act);
}
// MXFP8 variant: payloads are e4m3 bytes; `sfa` is the tiled scale tensor of the GATHERED A (every rank must
// hold all of it before the call, e.g. through an all-gather of the small scale tensors), `sfb` that of B.
int mt_ag_gemm_mxfp8(MtComm* c, void* stream, const void* const* a_shard, const void* const* sfa, const void* const* B,
                     const void* const* sfb, void* const* C, uint64_t gather_off, uint64_t flags_off, uint64_t epoch,
                     int M, int N, int K, int ldc, int ncomm, int nctas) {
  return ag_gemm_impl(c, stream, a_shard, B, C, gather_off, flags_off, epoch, M, N, K, ldc, ncomm, nctas, 0, 0, 1, true,
                      sfa, sfb);
}

// out[M / ranks, N] = reduce_scatter over rows of (A[M, K] * B[N, K]^T), K being this rank's slice of the
// contraction.  `stage_off`: symmetric buffer of 2 * ranks * (M / ranks) * N bf16 partial tiles.  Calls alternate
// between its halves (by the parity of `epoch`): a rank that has finished call e may already write partial tiles
// of call e + 1 into a peer whose reducers still read those of call e; it cannot reach call e + 2 before that
// peer has finished call e, because call e + 1 needs the peer's partial tiles of call e + 1.
// `flags_off`: symmetric u64 counters [ranks][M / ranks / 128][N / 256] followed by two ticket words, all zero
// before the first call.  `nred`: CTAs that only reduce (the others join them when their tiles are done).
static int gemm_rs_impl(MtComm* c, void* stream, const void* const* A, const void* const* B, void* const* out,
                        uint64_t stage_off, uint64_t flags_off, uint64_t epoch, int M, int N, int K, int nred, int nctas,
                        bool fp8, const void* const* sfa, const void* const* sfb, bool tb = false) {
  mt::GemmArgs a;
  if (fp8 && K % 128) return fail("MXFP8: K must be a multiple of 128");
  if (fused_common(c, a, M, N, K, flags_off, epoch)) return -1;
  int grid = nctas > 0 ? nctas : sm_count(c->device);
  if (c->emulated && grid * c->nlocal > sm_count(c->device)) grid = sm_count(c->device) / c->nlocal;
  if (nred < 0 || nred >= grid || (use_pair(M / c->nranks) && grid - ((nred + 1) & ~1) < 2)) return fail("nred out of range");
  if (c->nranks == 1) {
    // nothing to reduce: the product itself, without the staging area and the reducers' pass over it (8192 x 4096 x 1792:
    // 128 us with them, 83 without; stage_off, flags_off and epoch are not looked at).  The sum of one bf16 partial tile is
    // that tile.
    if ((uintptr_t)out[0] & 15) return fail("out must be 16-byte aligned");
    if (fp8 && (((uintptr_t)sfa[0] | (uintptr_t)sfb[0]) & 15)) return fail("scale tensors must be 16-byte aligned");
    if (tb)
      return gemm_pair(stream, A[0], nullptr, B[0], nullptr, out[0], M, N, K, N, nctas, false, mthost::ST_GEMM_RS, waits_of(a),
                       false, true);
    return gemm_plain(stream, A[0], fp8 ? sfa[0] : nullptr, B[0], fp8 ? sfb[0] : nullptr, out[0], M, N, K, N, nctas, fp8,
                      mthost::ST_GEMM_RS, waits_of(a));
  }
  if (tb && !use_pair(M / c->nranks)) return fail("a transposed B needs rows per rank that are a multiple of 256");
  a.ncomm = nred;
  a.ldc = N;
  a.stage_off = stage_off + (epoch & 1) * (uint64_t)M * N * 2;
  mt::GemmMaps maps;
  memset(&maps, 0, sizeof(maps));
  for (int lr = 0; lr < c->nlocal; ++lr) {
    a.c[lr] = out[lr];
    if (make_map(&maps.a[lr], A[lr], M, K, kBM, fp8) || make_map(&maps.b[lr], B[lr], N, K, kBN, fp8)) return -1;
    maps.a2[lr] = maps.a[lr];
    if ((uintptr_t)out[lr] & 15) return fail("out must be 16-byte aligned");
    if (fp8) {
      a.sfa[lr] = sfa[lr];
      a.sfb[lr] = sfb[lr];
    }
  }
  if (use_pair(M / c->nranks)) {
    mt::PairSfMaps sf;
    memset(&sf, 0, sizeof(sf));
    for (int lr = 0; lr < c->nlocal; ++lr) {
      if (tb ? make_map_t(&maps.b[lr], B[lr], K, N) : make_map(&maps.b[lr], B[lr], N, K, 128, fp8)) return -1;
      if (fp8 && (make_sf_map(&sf.sfa[lr], sfa[lr], (uint64_t)(M / 128) * (K / 128)) ||
                  make_sf_map(&sf.sfb[lr], sfb[lr], (uint64_t)(N / 128) * (K / 128))))
        return -1;
    }
    a.tb = tb;
    a.ncomm = (nred + 1) & ~1;
    const int nclusters = (grid - a.ncomm) / 2;
    cudaError_t e2 = mt::launch_gemm_pair(mt::MODE_GEMM_RS, maps, sf, a, nclusters, c->nlocal, (cudaStream_t)stream, fp8);
    if (e2 != cudaSuccess) return fail(std::string("pair gemm_rs launch: ") + cudaGetErrorString(e2));
    mthost::stat_add(mthost::ST_GEMM_RS, (uint64_t)(2.0 * M * N * K));
    return 0;
  }
  cudaError_t e = mt::launch_gemm_tc(mt::MODE_GEMM_RS, maps, a, grid, c->nlocal, (cudaStream_t)stream, fp8);
  if (e != cudaSuccess) return fail(std::string("gemm_rs launch: ") + cudaGetErrorString(e));
  mthost::stat_add(mthost::ST_GEMM_RS, (uint64_t)(2.0 * M * N * K));
  return 0;
}

int mt_gemm_rs(MtComm* c, void* stream, const void* const* A, const void* const* B, void* const* out,
               uint64_t stage_off, uint64_t flags_off, uint64_t epoch, int M, int N, int K, int nred, int nctas) {
  return gemm_rs_impl(c, stream, A, B, out, stage_off, flags_off, epoch, M, N, K, nred, nctas, false, nullptr, nullptr);
}
// The same with B stored [K, N] (the backward product of a column-parallel layer).
int mt_gemm_rs_t(MtComm* c, void* stream, const void* const* A, const void* const* B, void* const* out,
                 uint64_t stage_off, uint64_t flags_off, uint64_t epoch, int M, int N, int K, int nred, int nctas) {
  return gemm_rs_impl(c, stream, A, B, out, stage_off, flags_off, epoch, M, N, K, nred, nctas, false, nullptr, nullptr, true);
}
int mt_gemm_rs_mxfp8(MtComm* c, void* stream, const void* const* A, const void* const* sfa, const void* const* B,
                     const void* const* sfb, void* const* out, uint64_t stage_off, uint64_t flags_off, uint64_t epoch,
                     int M, int N, int K, int nred, int nctas) {
  return gemm_rs_impl(c, stream, A, B, out, stage_off, flags_off, epoch, M, N, K, nred, nctas, true, sfa, sfb);
}

// x (dtype 0 fp32, 1 fp16, 2 bf16; 16-byte aligned) -> e4m3 payload and one ue8m0 scale per 32 consecutive elements.
int mt_mxfp8_quantize(void* stream, int dtype, const void* x, void* data, void* scale, uint64_t nelems) {
  if (nelems % 32) return fail("MXFP8 tensors hold whole blocks of 32 elements");
  if (dtype < 0 || dtype > 2) return fail("MXFP8 quantisation takes fp32, fp16 and bf16");
  if (((uintptr_t)x | (uintptr_t)data) & 15) return fail("MXFP8 quantisation needs 16-byte aligned buffers");
  if (nelems == 0) return 0;
  cudaError_t e = mt::launch_mx_quant(dtype, x, data, scale, nelems, (cudaStream_t)stream);
  if (e != cudaSuccess) return fail(std::string("mxfp8 quantise launch: ") + cudaGetErrorString(e));
  return 0;
}

// Row-major scales [rows, K / 32] -> the tiled layout mt_gemm_mxfp8 reads (rows a multiple of 128, K of 128).
int mt_mxfp8_tile_scales(void* stream, const void* in, void* out, uint64_t rows, uint64_t kb) {
  if (rows % 128 || kb % 4 || rows / 128 > 65535 || kb / 4 > (1u << 30)) return fail("scales: rows a multiple of 128, K of 128");
  if (((uintptr_t)in | (uintptr_t)out) & 3) return fail("scales must be 4-byte aligned");
  if (rows == 0 || kb == 0) return 0;
  cudaError_t e = mt::launch_mx_tile(in, out, (uint32_t)(rows / 128), (uint32_t)(kb / 4), (cudaStream_t)stream);
  if (e != cudaSuccess) return fail(std::string("scale tiling launch: ") + cudaGetErrorString(e));
  return 0;
}

// Sum of MXFP8 tensors (e4m3 payload + ue8m0 scale per 32 elements) over all ranks.  op 0: all-reduce into
// (data_out_off, scale_out_off) of every rank; op 1: reduce-scatter, shard `rank` into the local outputs.
int mt_mxfp8_reduce(MtComm* c, void* stream, int op, uint64_t data_in_off, uint64_t scale_in_off,
                    uint64_t data_out_off, uint64_t scale_out_off, void* const* data_out, void* const* scale_out,
                    uint64_t nelems, int nctas) {
  if (!c || !c->d_comms) return fail("communicator is not finalized");
  if (nelems % 32) return fail("MXFP8 tensors hold whole blocks of 32 elements");
  const uint64_t nblocks = nelems / 32;
  if (op == mt::MX_REDUCESCATTER && nblocks % c->nranks) return fail("blocks must divide evenly over the ranks");
  if ((data_in_off | data_out_off) & 15) return fail("MXFP8 payloads must be 16-byte aligned");
  if (nctas < 1 || nctas > 148) return fail("nctas out of range");
  if (c->emulated && nctas * c->nlocal > 148) nctas = 148 / c->nlocal;
  mt::Mxfp8Args a;
  memset(&a, 0, sizeof(a));
  a.data_in_off = data_in_off;
  a.scale_in_off = scale_in_off;
  a.data_out_off = data_out_off;
  a.scale_out_off = scale_out_off;
  a.nblocks = nblocks;
  a.op = op;
  for (int lr = 0; lr < c->nlocal; ++lr) {
    a.data_out[lr] = data_out ? data_out[lr] : nullptr;
    a.scale_out[lr] = scale_out ? scale_out[lr] : nullptr;
  }
  cudaError_t e = mt::launch_mxfp8(c->d_comms, a, nctas, c->nlocal, (cudaStream_t)stream);
  if (e != cudaSuccess) return fail(std::string("mxfp8 launch: ") + cudaGetErrorString(e));
  mthost::stat_add(mthost::ST_MXFP8_REDUCE, nelems);
  return 0;
}

}  // extern "C"
