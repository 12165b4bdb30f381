// Geometry, descriptors and tensor maps shared by the corrector network's
// tensor-core kernels (k_conv.cu, k_wgrad.cu).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include "sclet_conv.cuh"
#include "sclet_tc.cuh"
#include "sclet_tc_ptx.cuh"

namespace sclet {
namespace conv {

constexpr int ROWS = 128;       // cells per tile
constexpr int MAX_STAGES = 3;   // tiles of input runs in flight
constexpr int SMEM_LIMIT = 226 * 1024;  // dynamic shared memory: 227 KB per CTA less the static part

// Shared-memory matrix descriptor without swizzle: lbo and sbo bytes.
// K-major: 8-row core matrices (rows 16 bytes apart) sbo apart, K chunks lbo
// apart.  MN-major: core matrices of 8 MN values (16 bytes) x 8 k (16 bytes
// apart), MN groups sbo apart, k groups lbo apart.
__device__ __forceinline__ uint64_t smem_desc_lin(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version
  return d;                // layout type 0: no swizzle
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          tc::smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(tc::smem_u32(bar))
      : "memory");
}

// tile -> (sample b, plane zh in 1..N, first slot s0 of the plane)
struct Tile {
  int b, zh, s0;
};
__device__ __forceinline__ Tile tile_of(int t, int N, int Np, int per_plane) {
  Tile x;
  const int j = t % per_plane;
  const int bz = t / per_plane;
  x.zh = 1 + bz % N;
  x.b = bz / N;
  x.s0 = Np + j * ROWS;
  return x;
}

// 2-D BF16 tensor map over an activation buffer as lines of 128 bytes (8 slots
// of 16 bytes), no swizzle, boxes of box_rows lines; lines outside the buffer
// read as zeros.
static inline cudaError_t make_map_lines(CUtensorMap *map, const void *ptr, long long lines, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return cudaErrorNotSupported;
  cuuint64_t dims[2] = {64, (cuuint64_t)lines};
  cuuint64_t strides[1] = {128};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace conv
}  // namespace sclet
