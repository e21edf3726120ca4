// Layout of the tensor-core contraction's A operand.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

namespace plx {
namespace {

constexpr int kBM = 256;          // rows of a tile
constexpr int kBK = 32;           // k of a tile (64 bytes of BF16: the 64-byte swizzle atom)

// The A operand (T, A0 or D^T split in BF16 high/low) is stored in the order
// the kernel reads it: [m-tile of 256 rows][k-slab of 32][256 rows][32 k], so
// every stage's tile (256 x 32) is one contiguous 16 KB block of HBM, and within
// the tile already in the shared-memory image the UMMA descriptors read: the
// 64-byte swizzle, in which the 16-byte chunk c of row r sits at chunk
// c ^ ((r >> 1) & 3) of its 64-byte row.  A stage's A tile is then one plain
// bulk copy.  Rows beyond n and k beyond n are zero.
__device__ __forceinline__ int64_t a_tile_pos(int64_t rr, int64_t kk) {
    return rr * kBK + ((((kk >> 3) ^ ((rr >> 1) & 3)) << 3) | (kk & 7));
}
__device__ __forceinline__ int64_t a_tiled(int64_t r, int64_t k, int64_t ktiles) {
    return ((r / kBM) * ktiles + k / kBK) * (int64_t)(kBM * kBK) + a_tile_pos(r % kBM, k % kBK);
}

__device__ __forceinline__ void split_store(double a, int64_t idx, __nv_bfloat16 *__restrict__ hi,
                                            __nv_bfloat16 *__restrict__ lo) {
    float x = (float)a;
    __nv_bfloat16 h = __float2bfloat16_rn(x);
    hi[idx] = h;
    lo[idx] = __float2bfloat16_rn(x - __bfloat162float(h));
}

}  // namespace
}  // namespace plx
