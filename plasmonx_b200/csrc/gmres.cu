// Batched complex GMRES in FP64 with the reference's semantics
// (src/solvers/gmres_module.f90:30-228), one independent Krylov space per
// column (frequency x polarisation), all columns advanced in lock step so that
// every Arnoldi step is ONE batched operator application.
//
// Per column, exactly as the reference: x0 = 0, v1 = b/||b||, Arnoldi with
// modified Gram-Schmidt for j < 25 and classical Gram-Schmidt with one
// re-orthogonalisation for j >= 25, Givens rotations with reference-BLAS
// zrotg/zrot semantics, the logged residual |g_{j+1}| compared with the
// absolute tolerance, then the triangular solve, x += V y and the true
// residual ||b - A x|| deciding convergence; no restart.
//
// Storage: Krylov vectors are kept in "slabs", one per step j, each holding
// the j-th basis vector of every column ([C][2][n] split complex), allocated
// when the step is reached so that memory follows the actual iteration count.
// The inner solves of a refinement may keep their basis in FP32 (half the
// projection traffic); dot products, Hessenberg, rotations and the iterate stay
// FP64, and the refinement's FP64 residual absorbs the storage rounding.
// Columns that converge leave the active list; the operator and the Arnoldi
// kernels only touch active columns.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <memory>
#include <type_traits>

#include "cpu_relax.h"
#include "pdl.cuh"
#include "plx_internal.h"

namespace plx {

namespace {

constexpr int kRows = 2048;     // rows per block in the Arnoldi kernels
constexpr int kThreads = 256;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block reduction of two doubles; result valid in thread 0.
__device__ __forceinline__ void block_sum2(double &a, double &b) {
    __shared__ double ra[32], rb[32];
    a = warp_sum(a);
    b = warp_sum(b);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) {
        ra[w] = a;
        rb[w] = b;
    }
    __syncthreads();
    if (w == 0) {
        int nw = blockDim.x >> 5;
        a = l < nw ? ra[l] : 0.0;
        b = l < nw ? rb[l] : 0.0;
        a = warp_sum(a);
        b = warp_sum(b);
    }
}

// The product's input split into BF16 high and low parts where it is formed (the
// tensor-core contraction's column rows), in place of a pass that reads it again.
__device__ __forceinline__ void split_column(const TcColumns &sp, int k, int r, double re, double im) {
    const float a = (float)re, b = (float)im;
    const __nv_bfloat16 ah = __float2bfloat16_rn(a), bh = __float2bfloat16_rn(b);
    auto *hi = reinterpret_cast<__nv_bfloat16 *>(sp.hi) + 2 * (int64_t)k * sp.ld + r;
    auto *lo = reinterpret_cast<__nv_bfloat16 *>(sp.lo) + 2 * (int64_t)k * sp.ld + r;
    hi[0] = ah;
    hi[sp.ld] = bh;
    lo[0] = __float2bfloat16_rn(a - __bfloat162float(ah));
    lo[sp.ld] = __float2bfloat16_rn(b - __bfloat162float(bh));
}

// X[k] = P[c] v elementwise for column c = act[k] of slab j (P = 1 when null): the
// input of a step's product.  Only for the first step and when columns have left
// the batch; otherwise `normalize_givens` has written it with the basis vector.
template <typename VT>
__global__ void gather_cols(int n, const int32_t *__restrict__ act, const VT *__restrict__ slab,
                            const double *__restrict__ P, double *__restrict__ X, TcColumns sp) {
    pdl_sync();
    const int k = blockIdx.y, c = act[k];
    const VT *src = slab + (int64_t)c * 2 * n;
    const double *p = P ? P + (int64_t)c * 2 * n : nullptr;
    double *dst = X + (int64_t)k * 2 * n;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        double re = (double)src[r], im = (double)src[n + r];
        if (p) {
            const double pr = p[r], pi = p[n + r], t = pr * re - pi * im;
            im = pr * im + pi * re;
            re = t;
        }
        dst[r] = re;
        dst[n + r] = im;
        if (sp.hi) split_column(sp, k, r, re, im);
    }
}

// Partial complex dots conj(V_i[c]) . W[k] for i in [i0, i1) over one chunk of
// kDotRows rows: every thread keeps kDotPT entries of W in registers and all
// eight warps work on every basis vector (warp reduction, then a fixed-order
// sum over the warps), so the kernel is bandwidth-bound for any number of
// basis vectors, including the single-vector projections of modified
// Gram-Schmidt.
constexpr int kDotPT = 4;
constexpr int kDotRows = kThreads * kDotPT;

template <typename VT>
__global__ void __launch_bounds__(kThreads) dots_partial(int n, int i0, int i1,
                                                         const int32_t *__restrict__ act,
                                                         VT *const *__restrict__ slabs,
                                                         const double *__restrict__ W,
                                                         double2 *__restrict__ part) {
    pdl_sync();
    __shared__ double2 red[kThreads / 32][32];
    const int k = blockIdx.y, c = act[k];
    const int r0 = blockIdx.x * kDotRows;
    const double *wr = W + (int64_t)k * 2 * n;
    double wre[kDotPT], wim[kDotPT];
#pragma unroll
    for (int q = 0; q < kDotPT; ++q) {
        int r = r0 + threadIdx.x + kThreads * q;
        wre[q] = r < n ? wr[r] : 0.0;
        wim[q] = r < n ? wr[n + r] : 0.0;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ni = i1 - i0;
    for (int g0 = 0; g0 < ni; g0 += 32) {
        const int gn = min(32, ni - g0);
        for (int t = 0; t < gn; ++t) {
            const VT *v = slabs[i0 + g0 + t] + (int64_t)c * 2 * n;
            double re = 0.0, im = 0.0;
#pragma unroll
            for (int q = 0; q < kDotPT; ++q) {
                int r = r0 + threadIdx.x + kThreads * q;
                if (r < n) {
                    double vr = (double)v[r], vi = (double)v[n + r];
                    re += vr * wre[q] + vi * wim[q];      // conj(v) * w
                    im += vr * wim[q] - vi * wre[q];
                }
            }
            re = warp_sum(re);
            im = warp_sum(im);
            if (lane == 0) red[warp][t] = make_double2(re, im);
        }
        __syncthreads();
        if (threadIdx.x < gn) {
            double2 s = make_double2(0.0, 0.0);
            for (int w = 0; w < kThreads / 32; ++w) {
                s.x += red[w][threadIdx.x].x;
                s.y += red[w][threadIdx.x].y;
            }
            part[((int64_t)k * gridDim.x + blockIdx.x) * ni + g0 + threadIdx.x] = s;
        }
        __syncthreads();
    }
}

// The same partial dots for projections onto eight or more basis vectors
// (classical Gram-Schmidt): the chunk of W is staged in shared memory once and
// each warp takes whole basis vectors, 32 rows per lane with the loads of 16
// rows in flight, so one warp reduction serves 1,024 rows of a vector (the
// kernel above pays one per 128 rows and keeps only 8 loads in flight a warp).
// Same chunking and partial layout as dots_partial.  A batch whose columns times
// row chunks leave SMs idle spreads the vectors over blockIdx.z (the sums are the
// same): 893 unknowns, 61 columns 47 -> 16 us a launch, 2,800 unknowns, 4
// columns (12 CTAs before) 86 -> 7.6 us.
template <typename VT>
__global__ void __launch_bounds__(kThreads) dots_wide(int n, int i0, int i1,
                                                      const int32_t *__restrict__ act,
                                                      VT *const *__restrict__ slabs,
                                                      const double *__restrict__ W,
                                                      double2 *__restrict__ part) {
    pdl_sync();
    __shared__ double wsh[2][kDotRows];
    const int k = blockIdx.y, c = act[k];
    const int r0 = blockIdx.x * kDotRows;
    const int rn = min(kDotRows, n - r0);
    const double *wr = W + (int64_t)k * 2 * n;
    for (int t = threadIdx.x; t < kDotRows; t += kThreads) {
        wsh[0][t] = t < rn ? wr[r0 + t] : 0.0;
        wsh[1][t] = t < rn ? wr[n + r0 + t] : 0.0;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ni = i1 - i0;
    for (int ii = warp + (kThreads / 32) * blockIdx.z; ii < ni; ii += (kThreads / 32) * gridDim.z) {
        const VT *v = slabs[i0 + ii] + (int64_t)c * 2 * n + r0;
        double re = 0.0, im = 0.0;
        constexpr int kBatch = 16;
        for (int q0 = 0; q0 < kDotRows / 32; q0 += kBatch) {
            VT vr[kBatch], vi[kBatch];
            if (rn == kDotRows) {
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    vr[q] = v[lane + 32 * (q0 + q)];
                    vi[q] = v[n + lane + 32 * (q0 + q)];
                }
            } else {
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    const int t = lane + 32 * (q0 + q);
                    vr[q] = t < rn ? v[t] : VT(0);
                    vi[q] = t < rn ? v[n + t] : VT(0);
                }
            }
#pragma unroll
            for (int q = 0; q < kBatch; ++q) {
                const int t = lane + 32 * (q0 + q);
                const double a = wsh[0][t], b = wsh[1][t];          // zero beyond rn
                re += (double)vr[q] * a + (double)vi[q] * b;        // conj(v) * w
                im += (double)vr[q] * b - (double)vi[q] * a;
            }
        }
        re = warp_sum(re);
        im = warp_sum(im);
        if (lane == 0) part[((int64_t)k * gridDim.x + blockIdx.x) * ni + ii] = make_double2(re, im);
    }
}

// Sums the chunk partials: h[k][ii] = sum_b part[k][b][ii]; optionally accumulates
// into H column j (Hcol[c][i0+ii] += h) when Hslab != nullptr.
__global__ void dots_finish(int nchunk, int ni, int i0, const int32_t *__restrict__ act,
                            const double2 *__restrict__ part, double2 *__restrict__ h,
                            double2 *__restrict__ Hcol, int hstride, int accumulate) {
    pdl_sync();
    int k = blockIdx.y;
    int ii = blockIdx.x * blockDim.x + threadIdx.x;
    if (ii >= ni) return;
    double2 s = make_double2(0.0, 0.0);
    for (int b = 0; b < nchunk; ++b) {
        double2 p = part[((int64_t)k * nchunk + b) * ni + ii];
        s.x += p.x;
        s.y += p.y;
    }
    h[(int64_t)k * ni + ii] = s;
    if (Hcol) {
        double2 *dst = Hcol + (int64_t)act[k] * hstride + i0 + ii;
        if (accumulate) {
            dst->x += s.x;
            dst->y += s.y;
        } else {
            *dst = s;
        }
    }
}

// W[k] -= sum_{ii} V_{i0+ii}[c] h[k][ii]   (sign = -1), or X[c] += ... (sign = +1,
// target indexed by column instead of compact position when by_col != 0).
//
// FIN: `h` holds the projections' chunk partials [k][ndot][ni], which every block
// sums itself (up to four chunks: a launch less); the first block of a column also
// adds them to H.
constexpr int kCombineFin = 4;
template <typename VT, bool FIN>
__device__ __forceinline__ void combine_setup(int n, int i0, int ni, int hld, int hoff, int k, int c,
                                              VT *const *__restrict__ slabs, const double2 *__restrict__ h, int ndot,
                                              double2 *__restrict__ Hcol, int hstride, int accumulate, double2 *sh,
                                              const VT **col) {
    for (int t = threadIdx.x; t < ni; t += blockDim.x) {
        double2 v;
        if (FIN) {
            v = make_double2(0.0, 0.0);
            for (int b = 0; b < ndot; ++b) {
                const double2 p = h[((int64_t)k * ndot + b) * hld + hoff + t];
                v.x += p.x;
                v.y += p.y;
            }
            if (blockIdx.x == 0) {
                double2 *dst = Hcol + (int64_t)c * hstride + i0 + t;
                *dst = accumulate ? make_double2(dst->x + v.x, dst->y + v.y) : v;
            }
        } else {
            v = h[(int64_t)k * hld + hoff + t];
        }
        sh[t] = v;
        col[t] = slabs[i0 + t] + (int64_t)c * 2 * n;
    }
    __syncthreads();
}

// Real and imaginary part of v h, and of conj(v) w, with the roundings the sums of the
// plain form have always had (one product rounded, the other fused): near the attainable
// accuracy its stopping test turns on the last bits of the iterate, so kernels that
// replace one another keep them, whatever the compiler would contract.  `whole`: the
// vector is one of the leading groups of eight, whose imaginary parts fuse vi h.x.
__device__ __forceinline__ double2 prod(double vr, double vi, double2 h, bool whole) {
    return make_double2(fma(vr, h.x, -__dmul_rn(vi, h.y)), whole ? fma(vi, h.x, __dmul_rn(vr, h.y))
                                                                 : fma(vr, h.y, __dmul_rn(vi, h.x)));
}
__device__ __forceinline__ double2 conj_prod(double vr, double vi, double wr, double wi) {
    return make_double2(fma(vr, wr, __dmul_rn(vi, wi)), fma(vr, wi, -__dmul_rn(vi, wr)));
}

// The FP64 basis (the plain form): every row is one chain over ii in ascending order.
// A block owns 32 rows: all 256 threads load 32 vectors of them and leave their
// products in shared memory, the next 32 vectors in flight, and two warps (re, im; a
// lane a row) add them in order.  A thread per row and all its loads left 44 CTAs at
// 2,800 unknowns and 4 columns (36 us a launch, now 12.6 us; 893 unknowns, 61 columns
// 27 -> 19 us).
constexpr int kChainRows = 32, kChainVec = 32;
constexpr size_t kChainSmem = 2 * kChainVec * 2 * kChainRows * sizeof(double);       // combine_chain's static part
template <bool FIN>
__global__ void __launch_bounds__(kThreads) combine_chain(int n, int i0, int ni, int hld, int hoff,
                                                          const int32_t *__restrict__ act,
                                                          double *const *__restrict__ slabs,
                                                          const double2 *__restrict__ h, int ndot, double sign,
                                                          double *__restrict__ Y, int by_col,
                                                          double2 *__restrict__ Hcol, int hstride, int accumulate) {
    pdl_sync();
    extern __shared__ double2 sh[];                       // ni coefficients, then ni column pointers
    __shared__ double ps[2][kChainVec][2][kChainRows];
    const double **col = reinterpret_cast<const double **>(sh + ni);
    const int k = blockIdx.y, c = act[k];
    combine_setup<double, FIN>(n, i0, ni, hld, hoff, k, c, slabs, h, ndot, Hcol, hstride, accumulate, sh, col);
    const int row = threadIdx.x % kChainRows, grp = threadIdx.x / kChainRows;
    const int r = blockIdx.x * kChainRows + row;
    const int rr = min(r, n - 1);                         // a valid row; its sum is not stored
    constexpr int G = kThreads / kChainRows, L = kChainVec / G;          // 8 groups, 4 vectors a thread
    double vr[L], vi[L];
    auto load = [&](int ii) {
#pragma unroll
        for (int q = 0; q < L; ++q) {
            const int t = ii + grp * L + q;
            vr[q] = t < ni ? col[t][rr] : 0.0;
            vi[q] = t < ni ? col[t][n + rr] : 0.0;
        }
    };
    double sum = 0.0;                                     // groups 0 and 1: re, im of the row
    load(0);
    int buf = 0;
    for (int ii = 0; ii < ni; ii += kChainVec, buf ^= 1) {
#pragma unroll
        for (int q = 0; q < L; ++q) {
            const int t = ii + grp * L + q;
            const double2 p = prod(vr[q], vi[q], t < ni ? sh[t] : make_double2(0.0, 0.0), t < (ni & ~7));
            ps[buf][grp * L + q][0][row] = p.x;
            ps[buf][grp * L + q][1][row] = p.y;
        }
        if (ii + kChainVec < ni) load(ii + kChainVec);
        __syncthreads();
        const int m = min(kChainVec, ni - ii);
        if (grp < 2) {
            if (m == kChainVec) {
#pragma unroll
                for (int q = 0; q < kChainVec; ++q) sum += ps[buf][q][grp][row];
            } else {
                for (int q = 0; q < m; ++q) sum += ps[buf][q][grp][row];
            }
        }
    }
    if (r >= n || grp >= 2) return;
    double *y = Y + (int64_t)(by_col ? c : k) * 2 * n + grp * n;
    y[r] += sign * sum;
}

// The FP32 basis of an inner solve: a block owns 256 / G rows of one column; its G
// groups of threads take every G-th basis vector each (loads of a batch of them in
// flight together) and the groups' sums are added in order.  G = 4 up to 16,384
// unknowns, where one thread per row leaves the chip idle whenever few columns are
// active, and 1 above, where a thread per row suffices.  G depends on n and ni alone,
// so a column's sums do not depend on its batch.  npart (optional): the sum of squares
// of the block's new rows.  13,528 unknowns, up to 21 columns and 256 vectors: 40 ->
// 22 us a launch on average.
template <int G, bool FIN>
__global__ void __launch_bounds__(kThreads) combine_inner(int n, int i0, int ni, int hld, int hoff,
                                                          const int32_t *__restrict__ act,
                                                          float *const *__restrict__ slabs,
                                                          const double2 *__restrict__ h, int ndot, double sign,
                                                          double *__restrict__ Y, int by_col, double *__restrict__ npart,
                                                          double2 *__restrict__ Hcol, int hstride, int accumulate) {
    pdl_sync();
    constexpr int RB = kThreads / G;
    extern __shared__ double2 sh[];                       // ni coefficients, then ni column pointers
    __shared__ double2 red[G > 1 ? kThreads : 1];
    const float **col = reinterpret_cast<const float **>(sh + ni);
    const int k = blockIdx.y, c = act[k];
    combine_setup<float, FIN>(n, i0, ni, hld, hoff, k, c, slabs, h, ndot, Hcol, hstride, accumulate, sh, col);
    const int row = threadIdx.x % RB, grp = threadIdx.x / RB;
    const int r = blockIdx.x * RB + row;
    const bool in = r < n;
    const int rr = in ? r : n - 1;                        // a valid row; its sum is not stored
    double ar = 0.0, ai = 0.0;
    constexpr int kBatch = 8;                             // basis vectors whose loads are in flight together
    int ii = grp;
    for (; ii + (kBatch - 1) * G < ni; ii += kBatch * G) {
        float vr[kBatch], vi[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            vr[q] = col[ii + q * G][rr];
            vi[q] = col[ii + q * G][n + rr];
        }
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            const double2 hh = sh[ii + q * G];
            ar += (double)vr[q] * hh.x - (double)vi[q] * hh.y;
            ai += (double)vr[q] * hh.y + (double)vi[q] * hh.x;
        }
    }
    for (; ii < ni; ii += G) {
        const float *v = col[ii];
        const double2 hh = sh[ii];
        const double vr = (double)v[rr], vi = (double)v[n + rr];
        ar += vr * hh.x - vi * hh.y;
        ai += vr * hh.y + vi * hh.x;
    }
    if (G > 1) {
        red[threadIdx.x] = make_double2(ar, ai);
        __syncthreads();
        if (grp == 0) {
#pragma unroll
            for (int g = 1; g < G; ++g) {
                ar += red[g * RB + row].x;
                ai += red[g * RB + row].y;
            }
        }
    }
    double sq = 0.0;
    if (in && grp == 0) {
        double *y = Y + (int64_t)(by_col ? c : k) * 2 * n;
        const double yr = y[r] + sign * ar, yi = y[n + r] + sign * ai;
        y[r] = yr;
        y[n + r] = yi;
        sq = yr * yr + yi * yi;
    }
    if (npart) {                                          // the same for the whole grid
        double dummy = 0.0;
        block_sum2(sq, dummy);
        if (threadIdx.x == 0) npart[(int64_t)k * gridDim.x + blockIdx.x] = sq;
    }
}

// Modified Gram-Schmidt of W[k] against V_0..V_j in one launch (n <= 4,096): one
// block per column keeps its rows of W in registers and walks the basis, the next
// vector's loads in flight during the block reduction of the current one.  256
// threads take kDotRows rows, as in dots_partial, and the sums run in its order
// (a thread's rows, the warp's lanes, the warps, the chunks), so both give the same
// bits.  The three short launches per vector it replaces (300 vectors over the first
// 24 steps) took 2.3-2.8 us each plus their gaps; now 11.7 us a step on average at 893
// unknowns.
template <int CHUNKS>
__global__ void __launch_bounds__(CHUNKS * kThreads) mgs_column(int n, int j, const int32_t *__restrict__ act,
                                                                double *const *__restrict__ slabs,
                                                                double *__restrict__ W, double2 *__restrict__ Hcol,
                                                                int hstride) {
    pdl_sync();
    constexpr int kWarps = kThreads / 32;
    __shared__ double2 red[2][CHUNKS][kWarps];
    const int k = blockIdx.x, c = act[k];
    const int chunk = threadIdx.x / kThreads, tid = threadIdx.x % kThreads;
    const int warp = tid >> 5, lane = tid & 31, r0 = chunk * kDotRows + tid;
    double *w = W + (int64_t)k * 2 * n;
    double wr[kDotPT], wi[kDotPT], vr[kDotPT], vi[kDotPT];
    auto load = [&](const double *src, double *re, double *im) {
#pragma unroll
        for (int q = 0; q < kDotPT; ++q) {
            const int r = r0 + q * kThreads;
            re[q] = r < n ? src[r] : 0.0;
            im[q] = r < n ? src[n + r] : 0.0;
        }
    };
    load(w, wr, wi);
    load(slabs[0] + (int64_t)c * 2 * n, vr, vi);
    for (int i = 0; i <= j; ++i) {
        double re = 0.0, im = 0.0;
#pragma unroll
        for (int q = 0; q < kDotPT; ++q) {
            const double2 p = conj_prod(vr[q], vi[q], wr[q], wi[q]);
            re += p.x;
            im += p.y;
        }
        double nr[kDotPT], ni[kDotPT];
        if (i < j) load(slabs[i + 1] + (int64_t)c * 2 * n, nr, ni);
        re = warp_sum(re);
        im = warp_sum(im);
        if (lane == 0) red[i & 1][chunk][warp] = make_double2(re, im);
        __syncthreads();
        double2 p = make_double2(0.0, 0.0);               // lane q: chunk q's sum over its warps
        if (lane < CHUNKS)
#pragma unroll
            for (int t = 0; t < kWarps; ++t) {
                p.x += red[i & 1][lane][t].x;
                p.y += red[i & 1][lane][t].y;
            }
        double2 h = make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < CHUNKS; ++q) {
            h.x += __shfl_sync(0xffffffffu, p.x, q);
            h.y += __shfl_sync(0xffffffffu, p.y, q);
        }
        if (threadIdx.x == 0) Hcol[(int64_t)c * hstride + i] = h;
#pragma unroll
        for (int q = 0; q < kDotPT; ++q) {
            const double2 p = prod(vr[q], vi[q], h, false);
            wr[q] -= p.x;
            wi[q] -= p.y;
            if (i < j) {
                vr[q] = nr[q];
                vi[q] = ni[q];
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kDotPT; ++q) {
        const int r = r0 + q * kThreads;
        if (r < n) {
            w[r] = wr[q];
            w[n + r] = wi[q];
        }
    }
}

// ||W[k]||_2 (dznrm2): partial sums of squares per chunk.
// Sum of squares of one chunk by a block of kThreads; valid in thread 0.
__device__ __forceinline__ double norm_chunk(int n, const double *__restrict__ w, int chunk) {
    int r0 = chunk * kRows, rn = min(kRows, n - r0);
    double s = 0.0, dummy = 0.0;
    for (int t = threadIdx.x; t < rn; t += kThreads) {
        double a = w[r0 + t], b = w[n + r0 + t];
        s += a * a + b * b;
    }
    block_sum2(s, dummy);
    return s;
}

__global__ void __launch_bounds__(kThreads) norm_partial(int n, const double *__restrict__ W,
                                                         double *__restrict__ part) {
    pdl_sync();
    const int k = blockIdx.y;
    const double s = norm_chunk(n, W + (int64_t)k * 2 * n, blockIdx.x);
    if (threadIdx.x == 0) part[(int64_t)k * gridDim.x + blockIdx.x] = s;
}

// `host`: the same norms in the run's words
__global__ void norm_finish(int nchunk, int count, const double *__restrict__ part,
                            double *__restrict__ out, double *__restrict__ host) {
    pdl_sync();
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    double s = 0.0;
    for (int b = 0; b < nchunk; ++b) s += part[(int64_t)k * nchunk + b];
    out[k] = sqrt(s);
    host[k] = sqrt(s);
}

// v_1 = b / ||b||; g_1 = ||b||; the slab's address into the table.
template <typename VT>
__global__ void start_vectors(int n, const int32_t *__restrict__ act, const double *__restrict__ nrm,
                              const double *__restrict__ B, VT *__restrict__ slab0, VT **__restrict__ slabs,
                              double2 *__restrict__ g, int gstride) {
    int k = blockIdx.y, c = act[k];
    if (blockIdx.x == 0 && k == 0 && threadIdx.x == 0) slabs[0] = slab0;
    double s = nrm[k];
    const double *b = B + (int64_t)c * 2 * n;
    VT *v = slab0 + (int64_t)c * 2 * n;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < 2LL * n;
         r += (int64_t)gridDim.x * blockDim.x)
        v[r] = (VT)(b[r] * (1.0 / s));
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        g[(int64_t)c * gstride] = make_double2(s, 0.0);
        for (int i = 1; i < gstride; ++i) g[(int64_t)c * gstride + i] = make_double2(0.0, 0.0);
    }
}

__device__ __forceinline__ double cabs_(double2 a) { return hypot(a.x, a.y); }

// x' = c x + s y, y' = c y - conj(s) x, with fixed roundings (see prod).
__device__ __forceinline__ void zrot_(double2 &x, double2 &y, double c, double2 s) {
    const double2 nx = make_double2(fma(c, x.x, fma(s.x, y.x, -__dmul_rn(s.y, y.y))),
                                    fma(c, x.y, fma(s.x, y.y, __dmul_rn(s.y, y.x))));
    const double2 ny = make_double2(fma(c, y.x, fma(-s.x, x.x, -__dmul_rn(s.y, x.y))),
                                    fma(c, y.y, fma(-s.x, x.y, __dmul_rn(s.y, x.x))));
    x = nx;
    y = ny;
}

__device__ __forceinline__ double2 shfl2(double2 v, int lane) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}
__device__ __forceinline__ double2 shfl_up2(double2 v, int o) {
    return make_double2(__shfl_up_sync(0xffffffffu, v.x, o), __shfl_up_sync(0xffffffffu, v.y, o));
}

// Givens update of column j by one warp (norm = H(j+1, j)).
// Hcol is the slab of H column j ([C][hstride] complex).
//
// The j earlier rotations form a chain: with a_0 = h_0 the i-th rotation gives
// h_i' = c_i a_i + s_i h_{i+1} and passes on a_{i+1} = c_i h_{i+1} - conj(s_i) a_i.
// One thread walking it in global memory paid a dependent load per rotation (81 us
// at 130 rotations, 94 us at 360).  A warp loads 32 rotations at a time, coalesced and
// a tile ahead.  SCAN (inner solves): the chain is a composition of maps a -> p a + q,
// composed with a 5-step scan; |p| <= 1 throughout, so that is as stable as the
// chain.  Otherwise (the plain form) every lane walks the chain in its order with
// the tile's values from shared memory, which keeps the chain's bits.
// The result depends on j alone, not on the batch.
struct Rotation {
    double2 s, h;
    double c;
};
// A column's part of H, the rotations and g, and the first tile of the chain.
struct GivensTile {
    double2 *h, *sn, *g;
    double *cs;
    double2 a, g0, g1, si, hn;
    double ci;
    __device__ GivensTile(int c, int lane, int j, double2 *Hcol, int hstride, double *cs_, double2 *sn_, double2 *g_,
                          int gstride, int cstride)
        : h(Hcol + (int64_t)c * hstride), sn(sn_ + (int64_t)c * cstride), g(g_ + (int64_t)c * gstride),
          cs(cs_ + (int64_t)c * cstride) {
        a = h[0];                            // chain value entering the tile (same in every lane)
        g0 = g[j];
        g1 = g[j + 1];
        ci = lane < j ? cs[lane] : 1.0;
        si = lane < j ? sn[lane] : make_double2(0.0, 0.0);
        hn = lane < j ? h[lane + 1] : make_double2(0.0, 0.0);
    }
};

// The rotation (c, s) that takes (ca, b), b >= 0, to (r, 0): c = |ca| / r, s = ca / |ca| b / r.
// Scaled by a power of two, with two reciprocal square roots; false where a square would leave
// the range (the general form follows).
__device__ __forceinline__ bool rotation(double2 ca, double b, double &cj, double2 &sj) {
    const double m = fmax(fmax(fabs(ca.x), fabs(ca.y)), b);
    if (!(m > 1e-290 && m < 1e290)) return false;
    const double f = __hiloint2double((2046 - ((__double2hiint(m) >> 20) & 0x7ff)) << 20, 0);   // 2^-exponent, or half
    const double x = ca.x * f, y = ca.y * f, z = b * f, a2 = fma(x, x, y * y);
    if (!(a2 > 1e-260)) return false;
    const double ia = rsqrt(a2), ir = rsqrt(fma(z, z, a2)), t = z * ir * ia;
    cj = a2 * ia * ir;
    sj = make_double2(x * t, y * t);
    return true;
}

template <bool SCAN>
__device__ void givens(int k, int lane, int j, double norm, const GivensTile &tile, double *__restrict__ resid,
                       Rotation *rot) {
    double2 *__restrict__ h = tile.h;
    double *__restrict__ csc = tile.cs;
    double2 *__restrict__ snc = tile.sn;
    double2 *__restrict__ gc = tile.g;
    double2 a = tile.a, g0 = tile.g0, g1 = tile.g1, si = tile.si, hn = tile.hn;
    double2 cb = make_double2(norm, 0.0);
    double ci = tile.ci;
    for (int i0 = 0; i0 < j; i0 += 32) {
        const int i = i0 + lane, in = i + 32;
        // the next tile's loads, in flight during this tile's chain
        const double cin = in < j ? csc[in] : 1.0;
        const double2 sin_ = in < j ? snc[in] : make_double2(0.0, 0.0);
        const double2 hnn = in < j ? h[in + 1] : make_double2(0.0, 0.0);
        if (SCAN) {
            double2 p = i < j ? make_double2(-si.x, si.y) : make_double2(1.0, 0.0);      // -conj(s)
            double2 q = i < j ? make_double2(ci * hn.x, ci * hn.y) : make_double2(0.0, 0.0);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double2 pp = shfl_up2(p, o), qq = shfl_up2(q, o);
                if (lane >= o) {
                    const double2 t = cmul(p, qq);
                    q.x += t.x;
                    q.y += t.y;
                    p = cmul(p, pp);
                }
            }
            const double2 t = cmul(p, a);
            const double2 out = make_double2(t.x + q.x, t.y + q.y);      // a after this lane's rotation
            double2 ai = shfl_up2(out, 1);                               // a before it
            if (lane == 0) ai = a;
            if (i < j)
                h[i] = make_double2(ci * ai.x + (si.x * hn.x - si.y * hn.y), ci * ai.y + (si.x * hn.y + si.y * hn.x));
            a = shfl2(out, 31);
        } else {
            __syncwarp();
            rot[lane] = Rotation{si, hn, ci};
            __syncwarp();
            const int m = min(32, j - i0);
            double2 mine = make_double2(0.0, 0.0);
#pragma unroll 8
            for (int t = 0; t < m; ++t) {
                const Rotation r = rot[t];
                double2 x = a, y = r.h;
                zrot_(x, y, r.c, r.s);
                if (lane == t) mine = x;
                a = y;
            }
            if (i < j) h[i] = mine;
        }
        ci = cin;
        si = sin_;
        hn = hnn;
    }
    if (lane != 0) return;
    double2 ca = a;
    double cj;
    double2 sj;
    if (SCAN && rotation(ca, norm, cj, sj)) {
    } else if (cabs_(ca) == 0.0) {
        cj = 0.0;
        sj = make_double2(1.0, 0.0);
    } else {
        double aa = cabs_(ca), ab = cabs_(cb);
        double scale = aa + ab;
        double2 cas = make_double2(ca.x / scale, ca.y / scale), cbs = make_double2(cb.x / scale, cb.y / scale);
        double t1 = cabs_(cas), t2 = cabs_(cbs);
        double norm = scale * sqrt(t1 * t1 + t2 * t2);
        double2 alpha = make_double2(ca.x / aa, ca.y / aa);
        cj = aa / norm;
        double2 s = cmul(alpha, cconj(cb));
        sj = make_double2(s.x / norm, s.y / norm);
    }
    csc[j] = cj;
    snc[j] = sj;
    zrot_(g0, g1, cj, sj);
    gc[j] = g0;
    gc[j + 1] = g1;
    zrot_(ca, cb, cj, sj);
    h[j] = ca;
    h[j + 1] = make_double2(0.0, 0.0);
    resid[k] = cabs_(g1);
}

// The end of an Arnoldi step: h_{j+1,j} = ||W[k]||, v_{j+1}[c] = W[k] / h_{j+1,j} (zero
// when the norm is zero, as the reference leaves the zero-filled column untouched),
// the Givens update of H's column j (one warp of a column's last block), and the
// input X[k] = P v_{j+1} of the next product, split for the tensor cores.  One launch
// in place of norm, scaling, Givens, gather, preconditioner and split.
//
// The norm: nparts partial sums of squares npart -- added by the block in the inner
// solves (VT float), in their order in the plain form -- or with nparts = 0 the chunks
// of W themselves (up to kNormChunks, in norm_partial's order).
//
// The launch also enters the new slab and H column in the address tables, which the
// kernels of the next steps read, and leaves the residual estimates in the run's words
// (take_words): three 8-byte copies in, one back and a clearing of the H column (every
// row that is read has been written) cost a step about 35 us of gaps between the kernels.
constexpr int kNormChunks = 2;
template <typename VT>
__global__ void __launch_bounds__(kThreads) normalize_givens(int n, int j, const int32_t *__restrict__ act, int nparts,
                                                             const double *__restrict__ npart,
                                                             const double *__restrict__ W, VT *__restrict__ slab_next,
                                                             const double *__restrict__ P, double *__restrict__ X,
                                                             TcColumns sp, VT **__restrict__ slabs,
                                                             double2 **__restrict__ Hcols, double2 *__restrict__ Hcol,
                                                             int hstride, double *__restrict__ cs,
                                                             double2 *__restrict__ sn, double2 *__restrict__ g,
                                                             int gstride, int cstride, double *__restrict__ resid) {
    pdl_sync();
    constexpr bool kInner = sizeof(VT) == 4;
    __shared__ double total;
    __shared__ Rotation rot[kInner ? 1 : 32];
    const int k = blockIdx.y, c = act[k];
    if (blockIdx.x == 0 && k == 0 && threadIdx.x == 0) {
        slabs[j + 1] = slab_next;
        Hcols[j] = Hcol;
    }
    // the last block of a column does its Givens update; its loads are in flight during
    // the norm, and so are the other blocks' first rows of W
    const bool last = blockIdx.x == gridDim.x - 1;
    const double *w = W + (int64_t)k * 2 * n;
    const int lane = threadIdx.x & 31, r0 = blockIdx.x * blockDim.x + threadIdx.x;
    const GivensTile tile(c, lane, last ? j : 0, Hcol, hstride, cs, sn, g, gstride, cstride);
    double wr = 0.0, wi = 0.0;
    if (!last && r0 < n) {
        wr = w[r0];
        wi = w[n + r0];
    }
    double s = 0.0;
    if (kInner) {
        double dummy = 0.0;
        for (int b = threadIdx.x; b < nparts; b += blockDim.x) s += npart[(int64_t)k * nparts + b];
        block_sum2(s, dummy);
    } else if (nparts == 0) {
        for (int q = 0; q * kRows < n; ++q) {
            const double p = norm_chunk(n, w, q);
            s += p;
        }
    } else if (threadIdx.x == 0) {
        for (int b = 0; b < nparts; ++b) s += npart[(int64_t)k * nparts + b];
    }
    if (threadIdx.x == 0) total = sqrt(s);
    __syncthreads();
    s = total;
    if (last) {
        if (threadIdx.x < 32) givens<kInner>(k, lane, j, s, tile, resid, rot);
        return;
    }
    const double inv = s != 0.0 ? 1.0 / s : 0.0;
    VT *v = slab_next + (int64_t)c * 2 * n;
    const double *p = P ? P + (int64_t)c * 2 * n : nullptr;
    double *x = X + (int64_t)k * 2 * n;
    for (int r = r0; r < n;) {
        const VT vr = (VT)(s != 0.0 ? wr * inv : 0.0), vi = (VT)(s != 0.0 ? wi * inv : 0.0);
        v[r] = vr;
        v[n + r] = vi;
        double re = (double)vr, im = (double)vi;
        if (p) {
            const double pr = p[r], pi = p[n + r], t = pr * re - pi * im;
            im = pr * im + pi * re;
            re = t;
        }
        x[r] = re;
        x[n + r] = im;
        if (sp.hi) split_column(sp, k, r, re, im);
        r += (gridDim.x - 1) * blockDim.x;
        if (r < n) {
            wr = w[r];
            wi = w[n + r];
        }
    }
}

// y = R^{-1} g for the triangular R = H(0..j, 0..j) (ztrsv 'U','N','N'), one block
// per triggered column, y stored compactly [k][j+1].  Back substitution in
// blocks of 32 columns: the 32 x 32 triangle lies in shared memory and is
// solved by one warp in registers, then the whole block subtracts the 32
// solved unknowns from the rows above (each row in descending column order and
// with the roundings of the unblocked substitution).  Those rows' entries (up to 256
// rows) and the next triangle are loaded into registers before the substitution
// starts, which left ~32 dependent multiplications a block: 31 us at 61-130 unknowns,
// 118 at 700, 7.9 at 20-60 (102, 333 and 18 us with the loads after it; 326 and 1,125
// by one warp with a dependent load per unknown).
constexpr int kTriB = 32;

// n / d rounded once from id = 1 / d rounded once (Markstein's theorem: the remainder
// of the first estimate is exact and its correction rounds correctly).
__device__ __forceinline__ double quotient(double n, double d, double id) {
    const double q = n * id;
    return fma(fma(-q, d, n), id, q);
}

constexpr int kTriThreads = 256;
__global__ void __launch_bounds__(kTriThreads) tri_solve(int count, int j, const int32_t *__restrict__ act,
                                                         double2 *const *__restrict__ Hcols, int hstride,
                                                         const double2 *__restrict__ g, int gstride,
                                                         double2 *__restrict__ y) {
    pdl_sync();
    extern __shared__ double2 ys[];
    __shared__ double2 tri[kTriB][kTriB + 1];        // tri[column][row]
    constexpr int kWarps = kTriThreads / 32, kCols = kTriB / kWarps;      // columns of a triangle a warp loads
    const int k = blockIdx.x;
    if (k >= count) return;
    const int c = act[k];
    const int m = j + 1;
    const int64_t off = (int64_t)c * hstride;
    const int warp = threadIdx.x >> 5, l = threadIdx.x & 31;
    const double2 zero = make_double2(0.0, 0.0);
    double2 next[kCols];                             // the next triangle, columns and rows b0 .. b0 + 31
    auto fetch = [&](int b0) {
#pragma unroll
        for (int q = 0; q < kCols; ++q) {
            const int col = warp + kWarps * q;
            next[q] = b0 + col < m && l <= col ? Hcols[b0 + col][off + b0 + l] : zero;
        }
    };
    auto store = [&] {
#pragma unroll
        for (int q = 0; q < kCols; ++q) tri[warp + kWarps * q][l] = next[q];
    };
    int b0 = (m - 1) / kTriB * kTriB;
    fetch(b0);
    for (int i = threadIdx.x; i < m; i += kTriThreads) ys[i] = g[(int64_t)c * gstride + i];
    store();
    __syncthreads();
    for (; b0 >= 0; b0 -= kTriB) {
        const int nb = min(kTriB, m - b0);
        // rows above and the next triangle, in flight during the substitution
        double2 r[kTriB];
#pragma unroll
        for (int q = 0; q < kTriB; ++q)
            r[q] = threadIdx.x < b0 && q < nb ? Hcols[b0 + q][off + threadIdx.x] : zero;
        if (b0 > 0) fetch(b0 - kTriB);
        if (warp == 0) {
            double2 v = l < nb ? ys[b0 + l] : zero;
            const double2 rd = l < nb ? tri[l][l] : make_double2(1.0, 0.0);
            const double d = fma(rd.x, rd.x, __dmul_rn(rd.y, rd.y)), id = 1.0 / d;
            for (int i = nb - 1; i >= 0; --i) {
                const double2 yi = shfl2(make_double2(quotient(fma(v.x, rd.x, __dmul_rn(v.y, rd.y)), d, id),
                                                      quotient(fma(v.y, rd.x, -__dmul_rn(v.x, rd.y)), d, id)),
                                         i);
                if (l == i) v = yi;
                if (l < i) {
                    const double2 p = prod(tri[i][l].x, tri[i][l].y, yi, false);
                    v.x -= p.x;
                    v.y -= p.y;
                }
            }
            if (l < nb) ys[b0 + l] = v;
        }
        __syncthreads();
        if (b0 > 0) {
            if (threadIdx.x < b0) {
                double2 v = ys[threadIdx.x];
#pragma unroll
                for (int q = kTriB - 1; q >= 0; --q)
                    if (q < nb) {
                        const double2 p = prod(r[q].x, r[q].y, ys[b0 + q], false);
                        v.x -= p.x;
                        v.y -= p.y;
                    }
                ys[threadIdx.x] = v;
            }
            for (int row = threadIdx.x + kTriThreads; row < b0; row += kTriThreads) {
                double2 v = ys[row];
                for (int i0 = nb; i0 > 0; i0 -= 8) {
                    double2 p[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) p[q] = i0 - 1 - q >= 0 ? Hcols[b0 + i0 - 1 - q][off + row] : zero;
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (i0 - 1 - q >= 0) {
                            const double2 t = prod(p[q].x, p[q].y, ys[b0 + i0 - 1 - q], false);
                            v.x -= t.x;
                            v.y -= t.y;
                        }
                }
                ys[row] = v;
            }
            store();
            __syncthreads();
        }
    }
    for (int i = threadIdx.x; i < m; i += kTriThreads) y[(int64_t)k * m + i] = ys[i];
}

// R[k] = B[c] - AX[k] with c = act[k]; in place into AX.
__global__ void residual(int n, const int32_t *__restrict__ act, const double *__restrict__ B,
                         double *__restrict__ AX) {
    pdl_sync();
    int k = blockIdx.y, c = act[k];
    const double *b = B + (int64_t)c * 2 * n;
    double *r = AX + (int64_t)k * 2 * n;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < 2LL * n;
         t += (int64_t)gridDim.x * blockDim.x)
        r[t] = b[t] - r[t];
}

__global__ void gather_x(int n, const int32_t *__restrict__ act, const double *__restrict__ X,
                         double *__restrict__ out) {
    pdl_sync();
    int k = blockIdx.y;
    const double *src = X + (int64_t)act[k] * 2 * n;
    double *dst = out + (int64_t)k * 2 * n;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < 2LL * n;
         r += (int64_t)gridDim.x * blockDim.x)
        dst[r] = src[r];
}

// Y[k] *= P[idx[k]] elementwise (complex), or in place on the column itself
// when by_col (Y indexed by idx[k]).
__global__ void scale_cols(int n, const int32_t *__restrict__ idx, const double *__restrict__ P,
                           double *__restrict__ Y, int by_col) {
    pdl_sync();
    int k = blockIdx.y, c = idx[k];
    const double *p = P + (int64_t)c * 2 * n;
    double *y = Y + (int64_t)(by_col ? c : k) * 2 * n;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
        double pr = p[r], pi = p[n + r], yr = y[r], yi = y[n + r];
        y[r] = pr * yr - pi * yi;
        y[n + r] = pr * yi + pi * yr;
    }
}

int grid_rows(int64_t n2) { return (int)std::min<int64_t>(n_blocks(n2, 256), 1024); }

// blockIdx.z of dots_wide() for `blocks` (row chunk, column) pairs and ni vectors: the
// fewest rounds of `slots` resident blocks (four an SM, two with an FP64 basis) times
// the vectors of a warp, half a vector for what a block does before them.  A split to a
// fixed number of blocks ran 784 of them as 1.3 rounds (13,528 unknowns, 14 columns, 120
// vectors: 40 us, now 35).
int dots_split(int blocks, int ni, int slots) {
    int best = 1;
    int64_t least = INT64_MAX;
    for (int nz = 1; nz <= std::min(64, n_blocks(ni, kThreads / 32)); ++nz) {
        const int64_t rounds = n_blocks((int64_t)blocks * nz, slots);
        const int64_t cost = rounds * (2 * n_blocks(ni, kThreads / 32 * nz) + 1);
        if (cost < least) {
            least = cost;
            best = nz;
        }
    }
    return best;
}

// Groups of threads of combine_inner() (see there).
int combine_groups(int n, int ni) { return n <= 16384 && ni >= 16 ? 4 : 1; }
int combine_blocks(int n, int ni) { return n_blocks(n, kThreads / combine_groups(n, ni)); }

// The basis combination over at most kCombine basis vectors per launch
// (shared-memory bound).  ndot > 0: h holds chunk partials (FIN), for ni <= kCombine.
// npart: norm partials of the last launch (FP32 basis).
constexpr int kCombine = 1024;
template <typename VT>
int64_t combine_chunked(cudaStream_t st, int sms, int n, int i0, int ni, int count, const int32_t *act,
                        VT *const *slabs, const double2 *h, double sign, double *Y, int by_col,
                        int ndot = 0, double *npart = nullptr, double2 *Hcol = nullptr, int hstride = 0,
                        int accumulate = 0) {
    int64_t launches = 0;
    for (int c0 = 0; c0 < ni; c0 += kCombine) {
        int cn = std::min(kCombine, ni - c0);
        // h is [count][ni]; pass the row stride through a shifted view per chunk
        const size_t smem = cn * (sizeof(double2) + sizeof(VT *));
        if constexpr (std::is_same<VT, double>::value) {
            const dim3 grid(n_blocks(n, kChainRows), count);
            // a few blocks an SM: unevenly spread they took 19.6 us at 2,800 unknowns x 4 columns, now 12.6
            const size_t even = even_smem((int64_t)grid.x * count, sms, kChainSmem, smem);
            launch_pdl((ndot ? combine_chain<true> : combine_chain<false>), grid, kThreads, even, st,
                       n, i0 + c0, cn, ni, c0, act, slabs, h, ndot, sign, Y, by_col, Hcol, hstride, accumulate);
        } else {
            const int G = combine_groups(n, ni);
            const dim3 grid(n_blocks(n, kThreads / G), count);
            double *np = c0 + cn == ni ? npart : nullptr;
#define PLX_COMBINE(GG, FIN)                                                                                    \
    launch_pdl(combine_inner<GG, FIN>, grid, kThreads, smem, st, n, i0 + c0, cn, ni, c0, act, slabs, h, ndot, sign, \
               Y, by_col, np, Hcol, hstride, accumulate)
            if (G == 4 && ndot) PLX_COMBINE(4, true);
            else if (G == 4) PLX_COMBINE(4, false);
            else if (ndot) PLX_COMBINE(1, true);
            else PLX_COMBINE(1, false);
#undef PLX_COMBINE
        }
        ++launches;
    }
    return launches;
}

}  // namespace

// Norms ||v[k]|| of a compact batch (used for ||b|| and the true residual).
static void batch_norms(plx_geom *g, int count, const double *V, DevArray<double> &part,
                        DevArray<double> &out, double *host) {
    plx_ctx *ctx = g->ctx;
    const int n = g->n_var;
    int nchunk = n_blocks(n, kRows);
    launch_pdl(norm_partial, dim3(nchunk, count), kThreads, 0, ctx->stream, n, V, part.p);
    launch_pdl(norm_finish, n_blocks(count, 128), 128, 0, ctx->stream, nchunk, count, part.p, out.p, host);
    ctx->launches += 2;
}

// One batched GMRES solve, advanced one Arnoldi step at a time so that the
// operator application of every step can be shared with other solves (a
// grouped tensor-core launch over several geometries): begin(), then while
// wants_product(): pre() -> the caller forms W = A X of the returned batch ->
// post() -> settle(); then end().  gmres_batched runs it with its own operator.
template <typename VT>
class GmresRun final : public GmresStepper {
  public:
    GmresRun(plx_geom *g, const GmresRequest &rq, const double *d_B, double *d_X, GmresResult &res)
        : g_(g), ctx_(g->ctx), st_(g->ctx->stream), rq_(rq), d_B_(d_B), d_X_(d_X), res_(res) {}

    void begin() {
        const int n = g_->n_var;
        C_ = (int)rq_.freq.size();
        m_ = std::min(rq_.m, n);
        res_.status.assign(C_, PLX_OK);
        res_.steps.assign(C_, 0);
        res_.trace.assign(rq_.record_trace ? (size_t)C_ * m_ : 0, 0.0);
        if (C_ == 0) return;
        if (m_ < 1) throw Error(PLX_ERR_ARG, "GMRES dimension must be positive");
        sms_ = sm_count(ctx_->device);
        nchunk_ = n_blocks(n, kRows);
        ndot_ = n_blocks(n, kDotRows);
        if ((size_t)(m_ + 1) * sizeof(double2) > 200 * 1024) throw Error(PLX_ERR_ARG, "GMRES dimension above 12800");
        once_per_device(reinterpret_cast<const void *>(tri_solve), ctx_->device, [] {
            PLX_CHECK_CUDA(cudaFuncSetAttribute(tri_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
            for (auto kern : {combine_chain<true>, combine_chain<false>})
                PLX_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 190 * 1024));
        });
        hstride_ = m_ + 1;   // rows of an H column (0..m)
        d_act_.alloc(ctx_, C_);
        d_freq_act_.alloc(ctx_, C_);
        d_cols_.alloc(ctx_, C_);
        Xa_.alloc(ctx_, (size_t)C_ * 2 * n);
        Wa_.alloc(ctx_, (size_t)C_ * 2 * n);
        work_.alloc(ctx_, (size_t)C_ * 2 * n);
        // norm partials: per kRows rows, or per block of combine()
        nrm_part_.alloc(ctx_, (size_t)C_ * std::max(nchunk_, n_blocks(n, kThreads / 4)));
        nrm_.alloc(ctx_, C_);
        cs_.alloc(ctx_, (size_t)C_ * m_);
        sn_.alloc(ctx_, (size_t)C_ * m_);
        gv_.alloc(ctx_, (size_t)C_ * hstride_);
        hbuf_.alloc(ctx_, (size_t)C_ * hstride_);
        ybuf_.alloc(ctx_, (size_t)C_ * hstride_);
        std::vector<DevArray<VT>>(m_ + 1).swap(slabs_);
        std::vector<DevArray<double2>>(m_).swap(hcols_);
        d_slabs_.alloc(ctx_, m_ + 1);
        d_hcols_.alloc(ctx_, m_);
        take_words();
        PLX_CHECK_CUDA(cudaMemsetAsync(d_X_, 0, (size_t)C_ * 2 * n * 8, st_));
        if (rq_.contraction == Contraction::TC3 || rq_.contraction == Contraction::TC1) split_ = tc_presplit(g_, C_);
        jac_ = rq_.jacobi && rq_.inner;
        if (jac_) {
            DevArray<int32_t> d_fall;
            d_fall.alloc(ctx_, C_);
            PLX_CHECK_CUDA(cudaMemcpyAsync(d_fall.p, rq_.freq.data(), C_ * 4, cudaMemcpyHostToDevice, st_));
            Pinv_.alloc(ctx_, (size_t)C_ * 2 * n);
            diagonal_inverse(g_, OpBatch{C_, d_fall.p}, Pinv_.p);
        }
        // active list: every column with ||b|| > 0 (the reference returns x = 0 otherwise)
        act_.resize(C_);
        for (int c = 0; c < C_; ++c) act_[c] = c;
        PLX_CHECK_CUDA(cudaMemcpyAsync(d_act_.p, act_.data(), C_ * 4, cudaMemcpyHostToDevice, st_));
        batch_norms(g_, C_, d_B_, nrm_part_, nrm_, words());   // B is [C] in column order == compact order here
        slabs_[0].alloc(ctx_, (size_t)C_ * 2 * n);
        start_vectors<VT><<<dim3(grid_rows(2LL * n), C_), 256, 0, st_>>>(n, d_act_.p, nrm_.p, d_B_, slabs_[0].p,
                                                                      d_slabs_.p, gv_.p, hstride_);
        ctx_->launches++;
        const double *bnorm = read_words(0, C_);
        act_.clear();
        for (int c = 0; c < C_; ++c) {
            if (!std::isfinite(bnorm[c])) {
                res_.status[c] = PLX_ERR_NAN;
            } else if (bnorm[c] > 0.0) {
                act_.push_back(c);
            }
        }
        upload_active();
        j_ = 0;
    }

    bool wants_product() const override { return C_ > 0 && j_ < m_ && !act_.empty(); }

    // w = A v_j for every active column: the batch the caller multiplies
    OpInput pre() override {
        const int n = g_->n_var;
        const int na = (int)act_.size();
        if (!x_ready_) {
            launch_pdl(gather_cols<VT>, dim3(grid_rows(n), na), 256, 0, st_, n, d_act_.p, slabs_[j_].p,
                       jac_ ? Pinv_.p : nullptr, Xa_.p, split_);
            ctx_->launches++;
        }
        return OpInput{g_, OpBatch{na, d_freq_act_.p}, Xa_.p, Wa_.p, work_.p, rq_.contraction, split_.hi != nullptr};
    }

    // launches the Arnoldi step on W and the least-squares update
    void post() override {
        const int n = g_->n_var;
        const int j = j_;
        const int na = (int)act_.size();
        hcols_[j].alloc(ctx_, (size_t)C_ * hstride_);
        slabs_[j + 1].alloc(ctx_, (size_t)C_ * 2 * n);
        size_t need = (size_t)na * ndot_ * (j + 1);
        if (part_.n < need) part_.alloc(ctx_, std::max(need, part_.n * 2));
        int nparts = 0;
        // W -= V V^H W over basis vectors i0..i1-1, the coefficients into (or added to) H's
        // column j; with an FP32 basis the last projection leaves the norm partials
        auto project = [&](int i0, int i1, int accumulate, bool last) {
            const int ni = i1 - i0;
            if (ni >= 8) {
                const int nz = dots_split(ndot_ * na, ni, (sizeof(VT) == 4 ? 4 : 2) * sms_);
                launch_pdl(dots_wide<VT>, dim3(ndot_, na, nz), kThreads, 0, st_, n, i0, i1, d_act_.p, d_slabs_.p,
                           Wa_.p, part_.p);
            } else {
                launch_pdl(dots_partial<VT>, dim3(ndot_, na), kThreads, 0, st_, n, i0, i1, d_act_.p, d_slabs_.p, Wa_.p,
                           part_.p);
            }
            ctx_->launches++;
            const bool fin = ndot_ <= kCombineFin && ni <= kCombine;
            if (!fin) {
                launch_pdl(dots_finish, dim3(n_blocks(ni, 128), na), 128, 0, st_, ndot_, ni, i0, d_act_.p, part_.p,
                           hbuf_.p, hcols_[j].p, hstride_, accumulate);
                ctx_->launches++;
            }
            if (last) nparts = combine_blocks(n, ni);
            ctx_->launches += combine_chunked(st_, sms_, n, i0, ni, na, d_act_.p, d_slabs_.p, fin ? part_.p : hbuf_.p, -1.0,
                                              Wa_.p, 0, fin ? ndot_ : 0, last ? nrm_part_.p : nullptr, hcols_[j].p,
                                              hstride_, accumulate);
        };
        prof_begin(ctx_);
        if (j + 1 < 25 && !rq_.inner) {
            if (!mgs_fused(na, j))
                for (int i = 0; i <= j; ++i) project(i, i + 1, 0, false);    // modified Gram-Schmidt
        } else {
            project(0, j + 1, 0, rq_.single_pass);                    // classical GS ...
            if (!rq_.single_pass) project(0, j + 1, 1, true);         // ... and re-orthogonalise
        }
        if (std::is_same<VT, double>::value) {
            nparts = 0;
            if (nchunk_ > kNormChunks) {
                launch_pdl(norm_partial, dim3(nchunk_, na), kThreads, 0, st_, n, Wa_.p, nrm_part_.p);
                ctx_->launches++;
                nparts = nchunk_;
            }
        }
        prof_end(ctx_, PROF_ORTHO, 0.0, 0.0);
        if (!host_.p) take_words();
        for (int k = 0; host_.p && k < na; ++k) memcpy(host_.p + k, &kPending, 8);
        prof_begin(ctx_);
        launch_pdl(normalize_givens<VT>, dim3(grid_rows(n) + 1, na), 256, 0, st_, n, j, d_act_.p, nparts, nrm_part_.p,
                   Wa_.p, slabs_[j + 1].p, jac_ ? Pinv_.p : nullptr, Xa_.p, split_, d_slabs_.p, d_hcols_.p,
                   hcols_[j].p, hstride_, cs_.p, sn_.p, gv_.p, hstride_, m_, words());
        ctx_->launches++;
        x_ready_ = true;
        prof_end(ctx_, PROF_LSQ, 0.0, 0.0);
        PLX_CHECK_CUDA(cudaGetLastError());
    }

    // waits for the step and tests its residuals
    void settle() override {
        const int n = g_->n_var;
        const int j = j_;
        const int na = (int)act_.size();
        const double *resid = await_residuals(na);
        std::vector<int32_t> trig;
        for (int k = 0; k < na; ++k) {
            int c = act_[k];
            res_.steps[c] = j + 1;
            if (rq_.record_trace) res_.trace[(size_t)c * m_ + j] = resid[k];
            const double tc = rq_.tols.empty() ? rq_.tol : rq_.tols[c];
            if (!std::isfinite(resid[k])) res_.status[c] = PLX_ERR_NAN;
            else if (resid[k] < tc || (rq_.inner && j == m_ - 1)) trig.push_back(c);
        }
        std::vector<char> done(C_, 0);
        for (int c : act_)
            if (res_.status[c] == PLX_ERR_NAN) done[c] = 1;
        if (!trig.empty() && rq_.inner) {
            // inner solve of a refinement: take the least-squares solution as is
            const int nt = (int)trig.size();
            PLX_CHECK_CUDA(cudaMemcpyAsync(d_cols_.p, trig.data(), nt * 4, cudaMemcpyHostToDevice, st_));
            launch_pdl(tri_solve, nt, kTriThreads, (j + 1) * sizeof(double2), st_, nt, j, d_cols_.p, d_hcols_.p,
                       hstride_, gv_.p, hstride_, ybuf_.p);
            ctx_->launches += 1 + combine_chunked(st_, sms_, n, 0, j + 1, nt, d_cols_.p, d_slabs_.p, ybuf_.p, 1.0, d_X_, 1);
            if (jac_) {
                launch_pdl(scale_cols, dim3(grid_rows(n), nt), 256, 0, st_, n, d_cols_.p, Pinv_.p, d_X_, 1);
                ctx_->launches++;
            }
            for (int c : trig) done[c] = 1;
            for (int c : trig)
                if (resid[std::find(act_.begin(), act_.end(), c) - act_.begin()] >=
                    (rq_.tols.empty() ? rq_.tol : rq_.tols[c]))
                    res_.status[c] = PLX_ERR_NOT_CONVERGED;   // inner dimension used up (not an error)
        } else if (!trig.empty()) {
            x_ready_ = false;                 // the true residual's product uses the input buffer
            const int nt = (int)trig.size();
            PLX_CHECK_CUDA(cudaMemcpyAsync(d_cols_.p, trig.data(), nt * 4, cudaMemcpyHostToDevice, st_));
            launch_pdl(tri_solve, nt, kTriThreads, (j + 1) * sizeof(double2), st_, nt, j, d_cols_.p, d_hcols_.p,
                       hstride_, gv_.p, hstride_, ybuf_.p);
            ctx_->launches += combine_chunked(st_, sms_, n, 0, j + 1, nt, d_cols_.p, d_slabs_.p, ybuf_.p, 1.0, d_X_, 1);
            launch_pdl(gather_x, dim3(grid_rows(2LL * n), nt), 256, 0, st_, n, d_cols_.p, d_X_, Xa_.p);
            ctx_->launches += 2;
            std::vector<int32_t> tf(nt);
            for (int t = 0; t < nt; ++t) tf[t] = rq_.freq[trig[t]];
            DevArray<int32_t> d_tf;
            d_tf.alloc(ctx_, nt);
            PLX_CHECK_CUDA(cudaMemcpyAsync(d_tf.p, tf.data(), nt * 4, cudaMemcpyHostToDevice, st_));
            OpBatch tb{nt, d_tf.p};
            apply_operator(g_, tb, Xa_.p, Wa_.p, work_.p,
                           Contraction::FP64 == rq_.contraction || Contraction::FP64_OTF == rq_.contraction
                               ? rq_.contraction
                               : Contraction::FP64);
            launch_pdl(residual, dim3(grid_rows(2LL * n), nt), 256, 0, st_, n, d_cols_.p, d_B_, Wa_.p);
            ctx_->launches++;
            batch_norms(g_, nt, Wa_.p, nrm_part_, nrm_, words() + C_);
            const double *tres = read_words(C_, nt);
            for (int t = 0; t < nt; ++t)
                if (tres[t] < rq_.tol) done[trig[t]] = 1;
                else if (!std::isfinite(tres[t])) {
                    res_.status[trig[t]] = PLX_ERR_NAN;
                    done[trig[t]] = 1;
                }
        }
        std::vector<int32_t> keep;
        for (int c : act_)
            if (!done[c]) keep.push_back(c);
        if (keep.size() != act_.size()) {
            act_.swap(keep);
            x_ready_ = false;                 // compact positions have changed
            if (!act_.empty()) upload_active();
        }
        ++j_;
    }

    void end() override {
        for (int c : act_) res_.status[c] = PLX_ERR_NOT_CONVERGED;
        act_.clear();
        PLX_CHECK_CUDA(cudaStreamSynchronize(st_));
    }

  private:
    // modified Gram-Schmidt in one launch where a block holds a column (the FP64 basis)
    bool mgs_fused(int na, int j) {
        if constexpr (std::is_same<VT, double>::value) {
            const int n = g_->n_var;
            if (n > 4 * kDotRows) return false;
#define PLX_MGS(Q)                                                                                             \
    launch_pdl(mgs_column<Q>, na, Q * kThreads, 0, st_, n, j, d_act_.p, d_slabs_.p, Wa_.p, hcols_[j].p, hstride_)
            if (n <= kDotRows) PLX_MGS(1);
            else if (n <= 2 * kDotRows) PLX_MGS(2);
            else PLX_MGS(4);
#undef PLX_MGS
            ctx_->launches++;
            return true;
        }
        return false;
    }

    // The residuals reach the host before the runtime reports the end of the kernel that
    // wrote them: reading the words for up to about ten milliseconds and then waiting
    // for the stream brings the next product forward: 9.8 -> 5.4 us after the step of a
    // matrix-free solve of 700 atoms, 12.2 -> 5.3 for six structures served together.
    // A residual with the pending word's bits costs that wait, nothing else.
    const double *await_residuals(int na) {
        if (!host_.p) {
            --ctx_->copy_steps;
            return read_words(0, na);
        }
        const volatile uint64_t *w = reinterpret_cast<const volatile uint64_t *>(host_.p);
        int k = 0;
        for (int polls = 0; k < na && polls < kPolls;) {
            if (w[k] != kPending) ++k;
            else {
                ++polls;
                cpu_relax();
            }
        }
        if (k < na) PLX_CHECK_CUDA(cudaStreamSynchronize(st_));
        std::atomic_thread_fence(std::memory_order_acquire);
        return host_.p;
    }

    // The words the kernels leave norms and residuals in: pinned host memory, or device
    // memory and a copy where none can be pinned (tried again kCopiedSteps steps later).
    void take_words() {
        const bool pin = ctx_->copy_steps <= 0;
        host_.alloc(ctx_, (size_t)2 * C_, pin);
        if (host_.p) return;
        if (pin) ctx_->copy_steps = kCopiedSteps;
        if (!dev_words_.p) {
            dev_words_.alloc(ctx_, (size_t)2 * C_);
            copy_.resize((size_t)2 * C_);
        }
    }
    double *words() { return host_.p ? host_.p : dev_words_.p; }
    // `count` words from `first`, written by kernels already launched
    const double *read_words(int first, int count) {
        if (!host_.p)
            PLX_CHECK_CUDA(cudaMemcpyAsync(copy_.data() + first, dev_words_.p + first, (size_t)count * 8,
                                           cudaMemcpyDeviceToHost, st_));
        PLX_CHECK_CUDA(cudaStreamSynchronize(st_));
        return (host_.p ? host_.p : copy_.data()) + first;
    }

    void upload_active() {
        std::vector<int32_t> fa(act_.size());
        for (size_t k = 0; k < act_.size(); ++k) fa[k] = rq_.freq[act_[k]];
        PLX_CHECK_CUDA(cudaMemcpyAsync(d_act_.p, act_.data(), act_.size() * 4, cudaMemcpyHostToDevice, st_));
        PLX_CHECK_CUDA(cudaMemcpyAsync(d_freq_act_.p, fa.data(), fa.size() * 4, cudaMemcpyHostToDevice, st_));
    }

    static constexpr uint64_t kPending = 0xfff8a5c35a3c0001ull;      // a NaN that no kernel forms
    static constexpr int kPolls = 1 << 18;

    plx_geom *g_;
    plx_ctx *ctx_;
    cudaStream_t st_;
    GmresRequest rq_;
    const double *d_B_;
    double *d_X_;
    GmresResult &res_;
    int sms_ = 1, C_ = 0, m_ = 0, j_ = 0, nchunk_ = 0, ndot_ = 0, hstride_ = 0;
    bool jac_ = false;
    TcColumns split_{nullptr, nullptr, 0};   // tensor-core runs: the split rows of the next input
    bool x_ready_ = false;      // Xa holds the next product's input
    std::vector<int32_t> act_;
    PinnedArray host_;          // residual estimates [C], true residuals [C]
    DevArray<double> dev_words_;             // the same without pinned memory,
    std::vector<double> copy_;               // and its copy
    DevArray<int32_t> d_act_, d_freq_act_, d_cols_;
    DevArray<double> Xa_, Wa_, work_, nrm_part_, nrm_, cs_, Pinv_;
    DevArray<double2> sn_, gv_, hbuf_, part_, ybuf_;
    std::vector<DevArray<VT>> slabs_;
    std::vector<DevArray<double2>> hcols_;
    DevArray<VT *> d_slabs_;
    DevArray<double2 *> d_hcols_;
};

std::unique_ptr<GmresStepper> make_gmres(plx_geom *g, const GmresRequest &rq, const double *d_B, double *d_X,
                                         GmresResult &res) {
    if (rq.inner && rq.basis_fp32) {
        auto r = std::make_unique<GmresRun<float>>(g, rq, d_B, d_X, res);
        r->begin();
        return r;
    }
    auto r = std::make_unique<GmresRun<double>>(g, rq, d_B, d_X, res);
    r->begin();
    return r;
}

void gmres_batched(plx_geom *g, const GmresRequest &rq, const double *d_B, double *d_X,
                   GmresResult &res) {
    auto run = make_gmres(g, rq, d_B, d_X, res);
    while (run->wants_product()) {
        OpInput in = run->pre();
        apply_operator(in.g, in.b, in.X, in.Y, in.work, in.how, in.presplit);
        run->post();
        run->settle();
    }
    run->end();
}

}  // namespace plx
