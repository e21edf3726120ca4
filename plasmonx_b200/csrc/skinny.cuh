// FP64 products S^T = X^T T with a stored row-major T: split over K into chunks
// whose partial sums are reduced in a fixed order.  Shared by the operator
// (operator.cu), the shifted Hessenberg solve and the no-allocation entry point
// (noalloc.cu).
#pragma once

#include <algorithm>
#include <cstdint>

#include "dmma.cuh"
#include "pdl.cuh"

namespace plx {
namespace {

constexpr int kSkinnyCols = 256;

// One warp computes 8 MT rows x 8 NT columns of a K chunk with the FP64 matrix
// instruction (dmma.cuh), its operands straight from global memory: every element
// of T is read by one warp of a row block, in 64-byte pieces, D steps of four k
// ahead in registers, so there is no shared memory and no barrier.  The block's
// four warps take WR row tiles and 4 / WR column tiles.
//
// With FMAs on the CUDA cores an operand from shared memory costs two cycles of the
// SM's one 128-byte port per warp, broadcast or not, against two cycles of one of
// its four FP64 pipes per FMA: 8 x 8 outputs a thread just balance (51-60% of the
// FP64 peak measured), one column a thread cannot (12 rows: 76% of the port, 18% of
// HBM).  The matrix instruction reads eight times fewer operands per FMA.
//   15,220 unknowns (T 1.85 GB): 6 rows 366 -> 281 us (6.6 TB/s), 12 rows 889 ->
//   366, 32 rows 1,098 -> 686, 42 rows 1,470 -> 863, 512 rows 12.4 -> 7.9 ms (30 TF).
// TR: the matrix is given by its transpose (T[k][col] lies at T[col * n + k]), read in
// 32-byte pieces; the sums are the same.  Rows beyond the batch and k beyond the chunk
// are zeros.  The order of an element's sum depends on n alone (skinny_split): not on R,
// MT, NT or its place.
template <int MT, int NT, int D, int WR, int MB, bool TR>
__global__ void __launch_bounds__(128, MB) product_partial(int R, int n, int kchunk, const double *__restrict__ Xt,
                                                           const double *__restrict__ T,
                                                           double *__restrict__ part) {
    pdl_sync();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kk = lane & 3, g = lane >> 2;
    const int col0 = (blockIdx.x * (4 / WR) + warp / WR) * 8 * NT, row0 = (blockIdx.y * WR + warp % WR) * 8 * MT;
    const int k0 = blockIdx.z * kchunk, k1 = min(n, k0 + kchunk);
    if (col0 >= n || row0 >= R) return;
    double acc[MT][NT][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
    double a[D][MT], b[D][NT];
    auto load = [&](int s, int k) {
        const bool in = k + kk < k1;
#pragma unroll
        for (int t = 0; t < NT; ++t)
            b[s][t] = in && col0 + 8 * t + g < n ? __ldg(TR ? T + (int64_t)(col0 + 8 * t + g) * n + k + kk
                                                            : T + (int64_t)(k + kk) * n + col0 + 8 * t + g)
                                                 : 0.0;
#pragma unroll
        for (int m = 0; m < MT; ++m)
            a[s][m] = in && row0 + 8 * m + g < R ? __ldg(Xt + (int64_t)(row0 + 8 * m + g) * n + k + kk) : 0.0;
    };
#pragma unroll
    for (int s = 0; s < D; ++s) load(s, k0 + 4 * s);
    for (int k = k0; k < k1; k += 4 * D) {
#pragma unroll
        for (int s = 0; s < D; ++s) {
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int t = 0; t < NT; ++t) dmma(acc[m][t], a[s][m], b[s][t]);
            load(s, k + 4 * D + 4 * s);
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const int r = row0 + 8 * m + g, c = col0 + 8 * t + 2 * kk;
            if (r < R) {
                double *o = part + ((int64_t)blockIdx.z * R + r) * n + c;
                if (c < n) o[0] = acc[m][t][0];
                if (c + 1 < n) o[1] = acc[m][t][1];
            }
        }
}

// Launches the partial products of R rows over ks chunks.  Row tiles: the fewest
// eights that hold the batch up to 48 rows (the fastest of the tilings tried at each
// size, 2 to 5 each at 7,844 and 15,220 unknowns); 32 rows a warp above, where
// the smaller tile's four blocks an SM beat 64 x 64 tiles (30 against 26 TF).
// Chunks of up to 16 k (up to 1,024 unknowns) end after one round of loads, so a warp's
// time is its latency and its stores, and 16 x 16 tiles, four times as many blocks, are
// faster until there are blocks enough without them.  Times with the sum, in those tiles
// against the ones above: 257 unknowns, 130 rows 11.7 against 16.0 us, 366 rows 19.6
// against 24.1; 800 unknowns, 32 rows 12.3 against 18.1, 48 rows 15.3 against 19.9 (the
// CUDA-core form, 34 rows: 14.9), 366 rows 82.5 against 74.2; 893 unknowns, 130 rows 33.7
// against 35.7, 366 rows 99 against 95; 1,400 unknowns (22 k), 130 rows 64 against 57.
template <bool TR = false>
void launch_product_partial(cudaStream_t st, int R, int n, int ks, int kchunk, const double *X, const double *T,
                            double *part) {
#define PLX_PP(MT, NT, D, WR, MB)                                                                                  \
    launch_pdl(product_partial<MT, NT, D, WR, MB, TR>,                                                                 \
               dim3((n + 32 / WR * NT - 1) / (32 / WR * NT), (R + 8 * MT * WR - 1) / (8 * MT * WR), ks), 128, 0, st, R, \
               n, kchunk, X, T, part)
    if (R <= 8) PLX_PP(1, 4, 4, 1, 1);
    else if (kchunk <= 16 && (int64_t)R * n <= 160000) PLX_PP(2, 2, 4, 2, 1);
    else if (R <= 16) PLX_PP(2, 4, 4, 1, 1);
    else if (R <= 24) PLX_PP(3, 4, 4, 1, 3);
    else if (R <= 32) PLX_PP(4, 4, 4, 1, 2);
    else if (R <= 48) PLX_PP(3, 8, 2, 2, 3);
    else PLX_PP(4, 4, 2, 2, 4);
#undef PLX_PP
}

__global__ void skinny_reduce(int n, int R, int ks, const double *__restrict__ part,
                              double *__restrict__ S) {
    pdl_sync();
    int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (int64_t)R * n) return;
    // the loads of eight partial sums together, added in order (64 of them one by one: 6.9 us
    // for 1,786 elements, now 5 us)
    const int64_t st = (int64_t)R * n;
    double s = 0.0;
    int k = 0;
    for (; k + 8 <= ks; k += 8) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = part[(k + q) * st + idx];
#pragma unroll
        for (int q = 0; q < 8; ++q) s += v[q];
    }
    for (; k < ks; ++k) s += part[k * st + idx];
    S[idx] = s;
}

// Number of K chunks and their length for a contraction of order n; depends on n only
// (592 blocks: four an SM of a B200, whatever the device), so that a column's sums depend
// neither on the batch it is part of nor on the device.
inline void skinny_split(int n, int &ks, int &kchunk) {
    const int cb = (n + kSkinnyCols - 1) / kSkinnyCols;
    ks = std::max(1, std::min(64, (592 + cb - 1) / cb));
    kchunk = (n + ks - 1) / ks;
    ks = (n + kchunk - 1) / kchunk;
}

}  // namespace
}  // namespace plx
