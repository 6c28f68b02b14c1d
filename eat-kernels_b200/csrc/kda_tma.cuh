// Tensor Memory Accelerator support: host-side tensor-map encoding (through the driver entry point, no link-time
// dependency on libcuda) and the device-side bulk tensor copy wrappers.
//
// Token tensors are described as rank-4 tensors {channel in a block, T (token), block, H (head)} with the caller's token
// stride, so a head slice of a wider tensor is read in place.  A block is 128 bytes of channels (64 bf16, 32 fp32), the row
// of the 128-byte swizzle; a tile is 32 tokens of one head, block after block in shared memory ([block][token][128 bytes]),
// and comes with ONE copy.  Rows past the end of the tensor are zero-filled by the hardware; rows past the end of a SEQUENCE
// belong to the next sequence and are masked by the consumers.  Every copy starts at channel 0 of block 0, the alignment the
// copy engine requires of the innermost coordinate.  No multicast is used anywhere.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace kda {

struct TmaMaps {
  CUtensorMap q, k, v, g;
};

inline int encode_token_map(CUtensorMap* map, const void* base, bool fp32, long long T, int H, long long ld_elems) {
  typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess || ptr == nullptr) return -1;
    fn = reinterpret_cast<EncodeFn>(ptr);
  }
  const int elem_bytes = fp32 ? 4 : 2, block_ch = 128 / elem_bytes, blocks = elem_bytes;      // 128 channels of a head
  const cuuint64_t dims[4] = {(cuuint64_t)block_ch, (cuuint64_t)T, (cuuint64_t)blocks, (cuuint64_t)H};
  const cuuint64_t strides[3] = {(cuuint64_t)ld_elems * elem_bytes, 128, (cuuint64_t)128 * elem_bytes};
  const cuuint32_t box[4] = {(cuuint32_t)block_ch, 32, (cuuint32_t)blocks, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUtensorMapDataType dt = fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const CUresult r = fn(map, dt, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(int)r - 1000;
}

#ifdef __CUDACC__
namespace tma {

__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" :: "r"(bar), "r"(bytes) : "memory");
}
// global -> shared copy of the tile of tokens [tok, tok + 32) of head h, completion (bytes) reported to the mbarrier
__device__ __forceinline__ void load_tile(uint32_t dst, const CUtensorMap* map, int h, int tok, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %2, %4}], [%5];\n"
               :: "r"(dst), "l"(map), "r"(0), "r"(tok), "r"(h), "r"(bar) : "memory");
}

}  // namespace tma
#endif

}  // namespace kda
