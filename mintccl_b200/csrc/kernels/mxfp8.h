// Arguments of the block-scaled fp8 reduction kernel.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "../device/layout.h"

namespace mt {
enum Mxfp8Op : int { MX_ALLREDUCE = 0, MX_REDUCESCATTER = 1 };
struct Mxfp8Args {
  void* data_out[MT_MAX_RANKS];   // reduce-scatter: local shard payload, per local rank
  void* scale_out[MT_MAX_RANKS];  // reduce-scatter: local shard scales
  uint64_t data_in_off, scale_in_off;    // heap offsets of the quantised input (every rank)
  uint64_t data_out_off, scale_out_off;  // all-reduce: heap offsets of the output (every rank)
  uint64_t nblocks;                      // 32-element blocks in the whole tensor
  int32_t op;
};
cudaError_t launch_mxfp8(const MtDevComm* comms, const Mxfp8Args& a, int nctas, int nlocal, cudaStream_t s);
// mxfp8_quant.cu: encoding (nelems a multiple of 32, x 16-byte aligned) and scale reordering (kq = K / 128 words a row)
cudaError_t launch_mx_quant(int dtype, const void* x, void* data, void* scale, uint64_t nelems, cudaStream_t s);
cudaError_t launch_mx_tile(const void* in, void* out, uint32_t row_blocks, uint32_t kq, cudaStream_t s);
}  // namespace mt
