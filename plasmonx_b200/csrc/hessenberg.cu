// Direct solve of the scalar-shift models through one Hessenberg reduction.
//
// For one-type wFQ (construct_dynamic_matrix_wfq, wfq_module.f90:214-254) and
// BEM DPCM (construct_dynamic_matrix_bem, bem_module.f90:881-933) the matrix
// complex_inversion factors at every frequency (algorithm_module.f90:510-541)
// is a real, frequency-independent A0 plus a complex multiple of the identity:
//     wFQ:   A(w) = (K - P) T - z(w) I          (one Drude z for every atom)
//     DPCM:  A(w) = D + z(w) I                  (z = 2 pi (eps_s + eps)/(eps_s - eps))
// so one orthogonal reduction A0 = Q H Q^T (H upper Hessenberg; Householder
// reflectors, backward stable) serves every frequency:
//     A(w) x = b   <=>   (H + s(w) I) y = Q^T b,   x = Q y,
// and each frequency costs O(n^2): Q^T b and Q y as dense products of the whole
// grid's right-hand sides with the explicit Q, and (H + s I) y = c by Givens
// rotations (QR of a Hessenberg matrix, no pivoting needed) and back
// substitution, one CTA per frequency (all its right-hand sides).  The result is
// the solution of the same linear system as the reference's zgetrf/zgetrs, to
// rounding (both factorisations are backward stable).
#include <algorithm>
#include <cmath>

#include "pdl.cuh"
#include "plx_internal.h"
#include "warp_sums.cuh"

namespace plx {

namespace {

constexpr int kT = 256;

// Sum over the block in a fixed order, in every thread; `red` holds a double per warp.
__device__ __forceinline__ double block_sum(double v, double *red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += red[k];
    return t;
}

// A0 of one-type wFQ, column-major: A0(r, c) = sum_e K_e (T[j_e][c] - T[r][c])
// (update_y_q of matrix_module.f90:1011-1098 applied to the columns of T).  A block takes one row and kT columns, so that a neighbour's row of T is
// read contiguously and its coefficient from shared memory; a thread per row, gathering
// down a column, took 1,024 us at 893 atoms, now 160 us.
__global__ void __launch_bounds__(kT) wfq_a0(int N, const int32_t *__restrict__ rowptr,
                                             const int32_t *__restrict__ col, const double *__restrict__ kval,
                                             const double *__restrict__ T, double *__restrict__ A) {
    __shared__ int32_t sj[kT];
    __shared__ double sk[kT];
    const int r = blockIdx.x, c = blockIdx.y * kT + threadIdx.x;
    const int cc = min(c, N - 1);
    const double trc = T[(int64_t)r * N + cc];
    double a = 0.0;
    for (int e0 = rowptr[r]; e0 < rowptr[r + 1]; e0 += kT) {
        const int m = min(kT, rowptr[r + 1] - e0);
        __syncthreads();
        if ((int)threadIdx.x < m) {
            sj[threadIdx.x] = col[e0 + threadIdx.x];
            sk[threadIdx.x] = kval[e0 + threadIdx.x];
        }
        __syncthreads();
        int q = 0;
        for (; q + 8 <= m; q += 8) {
            double t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) t[u] = T[(int64_t)sj[q + u] * N + cc];
#pragma unroll
            for (int u = 0; u < 8; ++u) a += sk[q + u] * (t[u] - trc);
        }
        for (; q < m; ++q) a += sk[q] * (T[(int64_t)sj[q] * N + cc] - trc);
    }
    if (c < N) A[(int64_t)c * N + r] = a;
}

// ---------------------------------------------------------------------------
// The reduction.  E = [A; Q] is column-major with 2 n rows: A in rows 0..n-1 and, below
// it, Q (the identity at the start), each an n x n array of its own: A becomes H and Q's
// array is Q^T row-major, so the reduction holds two matrices and leaves two.  Step k eliminates column k of A below its
// subdiagonal with the reflector I - beta v v^T:
//     A <- (I - beta v v^T) A (I - beta v v^T),   Q <- Q (I - beta v v^T).
// With y = E v and z = A^T v of the matrix before the step both sides are one
// rank-2 update of the columns right of k,
//     E_ij -= beta v_i z_j + beta u_i v_j,   u = y - beta (v^T y) v,   v = 0 in Q's rows,
// so a step is two launches: hh_gemv reads E once for y and z, hh_update reads
// and writes it once and leaves the norm of the next column.  Row and column
// tiles give fixed-order partial sums (at most ~28 each way).
//
// Bound by the chain of 2 (n - 2) dependent short launches up to a few thousand
// unknowns (E stays in L2), by HBM above.  The four-launch form (vector, left
// update, A v with a thread per row over all columns, right update) spent 113 of
// its 122 us a step at 893 unknowns in A v on 4 CTAs: 108.3 ms for the reduction,
// now 11.0 ms.
// ---------------------------------------------------------------------------
constexpr int kHR = 64, kHC = 32;          // rows and columns a block's inner tile holds

struct HessTiles {
    int n, rt, ct, nrc, ncc;               // rows and columns a block, number of row and column tiles
};
// Row i of [A; Q]: its element in column j lies j n further on.
template <typename P>
__device__ __forceinline__ P e_row(P A, P Q, int n, int i) {
    return i < n ? A + i : Q + (i - n);
}

HessTiles hess_tiles(int n) {
    HessTiles t;
    t.n = n;
    t.rt = kHR * std::max(1, (n_blocks(2 * n, kHR) + 27) / 28);
    t.ct = kHC * std::max(1, (n_blocks(n, kHC) + 27) / 28);
    t.nrc = n_blocks(2 * n, t.rt);
    t.ncc = n_blocks(n, t.ct);
    return t;
}

// Sum of squares of column 0 below its subdiagonal, per row tile.
__global__ void hh_norm0(HessTiles t, const double *__restrict__ A, double *__restrict__ npart) {
    __shared__ double red[kT / 32];
    double s = 0.0;
    for (int i = blockIdx.x * t.rt + threadIdx.x; i < min(t.n, (int)(blockIdx.x + 1) * t.rt); i += blockDim.x)
        if (i >= 2) s += A[i] * A[i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) npart[blockIdx.x] = s;
}

// y and z partial sums of step k over one tile, and v^T (tile) v.  Every block
// forms the reflector itself from column k (which no later step changes) and the
// column's norm; the first column tile's blocks store it.
__global__ void __launch_bounds__(kT) hh_gemv(HessTiles t, int k, int c0, const double *__restrict__ A,
                                              const double *__restrict__ Q,
                                              const double *__restrict__ npart, double *__restrict__ vbuf,
                                              double *__restrict__ beta, double *__restrict__ sub,
                                              double *__restrict__ yp, double *__restrict__ zp,
                                              double *__restrict__ sp) {
    pdl_sync();
    extern __shared__ double sm[];
    __shared__ double red[kT / 32], yred[kT / kHR][kHR];
    double *vr = sm, *vc = vr + t.rt, *zs = vc + t.ct;        // rt, ct, 2 ct
    const int n = t.n;
    const int cc = c0 + blockIdx.x, rc = blockIdx.y;
    const int i0 = rc * t.rt, i1 = min(2 * n, i0 + t.rt);
    const int j0 = cc * t.ct, j1 = min(n, j0 + t.ct);
    const double *ck = A + (int64_t)k * n;
    const double x0 = ck[k + 1];
    double tail = 0.0;                                        // the same in every warp
    for (int r = threadIdx.x & 31; r < t.nrc; r += 32) tail += npart[r];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tail += __shfl_xor_sync(0xffffffffu, tail, o);
    const double nrm = sqrt(x0 * x0 + tail);
    const bool none = nrm == 0.0 || tail == 0.0;              // nothing to eliminate: identity
    const double alpha = none ? x0 : (x0 >= 0.0 ? -nrm : nrm);
    const double v0 = x0 - alpha;
    const double b = none ? 0.0 : 2.0 / (v0 * v0 + tail);
    auto v_of = [&](int i) { return none || i <= k || i >= n ? 0.0 : (i == k + 1 ? v0 : ck[i]); };
    for (int i = threadIdx.x; i < t.rt; i += kT) vr[i] = v_of(i0 + i);
    for (int j = threadIdx.x; j < t.ct; j += kT) {
        vc[j] = v_of(j0 + j);                                 // zero for columns <= k
        zs[j] = zs[t.ct + j] = 0.0;
    }
    __syncthreads();
    if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i < t.rt; i += kT)
            if (i0 + i < n) vbuf[i0 + i] = vr[i];
        if (rc == 0 && threadIdx.x == 0) {
            beta[0] = b;
            sub[k] = alpha;
        }
    }
    const int row = threadIdx.x % kHR, cg = threadIdx.x / kHR, lane = threadIdx.x & 31, half = (row >> 5) & 1;
    constexpr int NC = kHC / (kT / kHR);                      // columns a thread in the inner tile: 8
    for (int rs = 0; i0 + rs < i1; rs += kHR) {
        const int i = i0 + rs + row;
        const double *e = e_row(A, Q, n, i);
        const bool in = i < i1, left = i0 + rs < n && i0 + rs + kHR > k + 1;
        const double vi = vr[rs + row];
        double y = 0.0;
        for (int cs = 0; j0 + cs < j1; cs += kHC) {
            double a[NC];
#pragma unroll
            for (int q = 0; q < NC; ++q) {
                const int j = j0 + cs + cg * NC + q;
                a[q] = in && j < j1 && j > k ? e[(int64_t)j * n] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < NC; ++q) {
                y = fma(a[q], vc[cs + cg * NC + q], y);
                a[q] *= vi;
            }
            if (left) {
                const int q = lane_sums<NC>(a, lane);
                if (lane % (32 / NC) == 0) zs[half * t.ct + cs + cg * NC + q] += a[0];
            }
        }
        yred[cg][row] = y;
        __syncthreads();
        if (threadIdx.x < kHR && in) {
            double s = 0.0;
            for (int c = 0; c < kT / kHR; ++c) s += yred[c][row];
            yp[(int64_t)cc * 2 * n + i] = s;
        }
        __syncthreads();
    }
    double s = 0.0;
    for (int j = threadIdx.x; j < t.ct; j += kT)
        if (j0 + j < j1) {
            const double z = zs[j] + zs[t.ct + j];
            zp[(int64_t)rc * n + j0 + j] = z;
            s += z * vc[j];
        }
    s = block_sum(s, red);
    if (threadIdx.x == 0) sp[rc * t.ncc + cc] = s;
}

// The rank-2 update of one tile, and the partial norm of column k + 1 below its
// subdiagonal from the blocks that hold it.
__global__ void __launch_bounds__(kT) hh_update(HessTiles t, int k, int c0, double *__restrict__ A,
                                                double *__restrict__ Q,
                                                const double *__restrict__ vbuf, const double *__restrict__ beta,
                                                const double *__restrict__ yp, const double *__restrict__ zp,
                                                const double *__restrict__ sp, double *__restrict__ npart) {
    pdl_sync();
    extern __shared__ double sm[];
    __shared__ double red[kT / 32];
    // rt, rt, ct, ct, and the partial sums' sums: 4 rt, 8 ct
    double *bv = sm, *bu = bv + t.rt, *vc = bu + t.rt, *zc = vc + t.ct, *yq = zc + t.ct, *zq = yq + 4 * t.rt;
    const int n = t.n;
    const int cc = c0 + blockIdx.x, rc = blockIdx.y;
    const int i0 = rc * t.rt, i1 = min(2 * n, i0 + t.rt);
    const int j0 = cc * t.ct, j1 = min(n, j0 + t.ct);
    const int row = threadIdx.x % kHR, cg = threadIdx.x / kHR;
    constexpr int NC = kHC / (kT / kHR);
    double first[NC];                                         // the first inner tile, in flight from here
    const double *e0 = e_row(A, Q, n, i0 + row);
#pragma unroll
    for (int q = 0; q < NC; ++q) {
        const int j = j0 + cg * NC + q;
        first[q] = i0 + row < i1 && j < j1 && j > k ? e0[(int64_t)j * n] : 0.0;
    }
    const double b = beta[0];
    const int nra = (n + t.rt - 1) / t.rt;                    // row tiles that hold rows of A
    double s = 0.0;
    for (int e = threadIdx.x; e < nra * (t.ncc - c0); e += kT)
        s += sp[e / (t.ncc - c0) * t.ncc + c0 + e % (t.ncc - c0)];
    for (int i = row; i < t.rt; i += kHR) {                   // four threads a row
        double y = 0.0;
        if (i0 + i < i1)
#pragma unroll 8
            for (int c = c0 + cg; c < t.ncc; c += kT / kHR) y += yp[(int64_t)c * 2 * n + i0 + i];
        yq[cg * t.rt + i] = y;
    }
    for (int j = threadIdx.x % kHC; j < t.ct; j += kHC) {     // eight threads a column
        double z = 0.0;
        if (j0 + j < j1)
#pragma unroll 4
            for (int r = threadIdx.x / kHC; r < nra; r += kT / kHC) z += zp[(int64_t)r * n + j0 + j];
        zq[threadIdx.x / kHC * t.ct + j] = z;
    }
    s = b * block_sum(s, red);
    for (int i = threadIdx.x; i < t.rt; i += kT) {
        const double y = (yq[i] + yq[t.rt + i]) + (yq[2 * t.rt + i] + yq[3 * t.rt + i]);
        const double v = i0 + i < n ? vbuf[i0 + i] : 0.0;
        bv[i] = b * v;
        bu[i] = b * (y - s * v);
    }
    for (int j = threadIdx.x; j < t.ct; j += kT) {
        double z = 0.0;
        for (int r = 0; r < kT / kHC; ++r) z += zq[r * t.ct + j];
        vc[j] = j0 + j < j1 ? vbuf[j0 + j] : 0.0;
        zc[j] = z;
    }
    __syncthreads();
    const bool next = j0 <= k + 1 && k + 1 < j1;
    double sq = 0.0;
    for (int rs = 0; i0 + rs < i1; rs += kHR) {
        const int i = i0 + rs + row;
        if (i >= i1) continue;
        double *e = e_row(A, Q, n, i);
        const double v = bv[rs + row], u = bu[rs + row];
        for (int cs = 0; j0 + cs < j1; cs += kHC) {
            double a[NC];
#pragma unroll
            for (int q = 0; q < NC; ++q) {
                const int j = j0 + cs + cg * NC + q;
                a[q] = rs + cs == 0 ? first[q] : (j < j1 && j > k ? e[(int64_t)j * n] : 0.0);
            }
#pragma unroll
            for (int q = 0; q < NC; ++q) {
                const int j = j0 + cs + cg * NC + q;
                if (j < j1 && j > k) {
                    const double x = a[q] - (v * zc[cs + cg * NC + q] + u * vc[cs + cg * NC + q]);
                    e[(int64_t)j * n] = x;
                    if (j == k + 1 && i >= k + 3 && i < n) sq += x * x;
                }
            }
        }
    }
    if (next) {                                               // the same for the whole block
        sq = block_sum(sq, red);
        if (threadIdx.x == 0) npart[rc] = sq;
    }
}

__global__ void hess_identity(int n, double *__restrict__ Q) {
    const int j = blockIdx.y;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        Q[(int64_t)j * n + i] = i == j ? 1.0 : 0.0;
}

// The reduced A, column-major, to H row-major (the rows the Givens sweep reads) in
// place, upper Hessenberg part: a block exchanges two mirrored 32 x 32 tiles.
__global__ void hess_rows(int n, double *__restrict__ A, const double *__restrict__ sub) {
    if (blockIdx.x < blockIdx.y) return;
    __shared__ double tile[2][32][33];                        // rows of block x, columns of block y; the mirror
    const int b[2] = {(int)blockIdx.x * 32, (int)blockIdx.y * 32};
    for (int m = 0; m < 2; ++m)
        for (int y = threadIdx.y; y < 32; y += blockDim.y) {
            const int r = b[m] + threadIdx.x, c = b[1 - m] + y;
            if (r >= n || c >= n) continue;
            const double a = A[(int64_t)c * n + r];
            tile[m][y][threadIdx.x] = c >= r ? a : (c == r - 1 ? (c + 2 < n ? sub[c] : a) : 0.0);
        }
    __syncthreads();
    for (int m = 0; m < 2; ++m)                               // (on the diagonal both are the same tile)
        for (int y = threadIdx.y; y < 32; y += blockDim.y) {
            const int r = b[m] + y, c = b[1 - m] + threadIdx.x;
            if (r < n && c < n) A[(int64_t)r * n + c] = tile[m][threadIdx.x][y];
        }
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

// One frequency per block: solves (H + s I) y = c for each of its `cols`
// right-hand sides (split complex [2][n] in C, in place).  R (the triangular
// factor, rows packed, n (n + 1) / 2 complex) lives in this block's slice of Rbuf;
// the carry row and y in shared memory (dynamic: (1 + cols) n complex).
//
// Latency bound: n dependent rotations, then n / 32 blocks of back substitution,
// with one CTA per frequency and 61 frequencies far from filling the chip.  So a
// step of the sweep has one barrier: every thread forms the rotation itself (step k
// writes no carry[k], which all threads read), and the next row of H is loaded a
// step ahead.
// The back substitution solves 32 unknowns in one warp and subtracts them from
// the rows above a warp per row.  893 unknowns, 61 frequencies, 3 columns: the
// former sweep and the reflectors applied one by one took 10.7 ms, now 1.9 ms with the two products.
constexpr int kSolveT = 512;
constexpr int kAhead = 4;            // elements of the next row a thread loads ahead

__device__ __forceinline__ void rotation(double2 a, double b, double &c, double2 &sn) {
    // zrotg on (a, b), b real: c real, sn = (a / |a|) b / |(a, b)|
    double aa2 = a.x * a.x + a.y * a.y, m = aa2 + b * b;
    if (aa2 > 1e-290 && m < 1e290) {
        const double ia = rsqrt(aa2), in = rsqrt(m);
        const double f = ia * in * b;
        c = aa2 * ia * in;
        sn = make_double2(a.x * f, a.y * f);
        return;
    }
    const double aa = hypot(a.x, a.y);
    if (aa == 0.0) {
        c = 0.0;
        sn = make_double2(1.0, 0.0);
        return;
    }
    const double nr = hypot(aa, b);
    c = aa / nr;
    sn = make_double2(a.x / aa * (b / nr), a.y / aa * (b / nr));
}

__global__ void __launch_bounds__(kSolveT) hess_solve(int n, int cols, const int32_t *__restrict__ freq_of_block,
                                                      const Cplx *__restrict__ shift, const double *__restrict__ Hr,
                                                      double *__restrict__ C, double2 *__restrict__ Rbuf,
                                                      int *__restrict__ singular) {
    extern __shared__ double2 sh[];
    __shared__ double2 tri[32][33];     // tri[column][row] of a diagonal block of R
    const int blk = blockIdx.x;
    const Cplx sv = shift[freq_of_block[blk]];
    const double2 s = make_double2(sv.re, sv.im);
    double2 *carry = sh;                // n
    double2 *y = sh + n;                // cols x n
    double2 *R = Rbuf + (int64_t)blk * ((int64_t)n * (n + 1) / 2);
    double *Cb = C + (int64_t)blk * cols * 2 * n;
    for (int c = 0; c < cols; ++c)
        for (int i = threadIdx.x; i < n; i += kSolveT)
            y[(int64_t)c * n + i] = make_double2(Cb[(int64_t)c * 2 * n + i], Cb[(int64_t)c * 2 * n + n + i]);
    // Givens QR of (H + s I): carry row 0, then rotate it against rows 1..n-1
    for (int j = threadIdx.x; j < n; j += kSolveT)
        sh[j] = make_double2(Hr[j] + (j == 0 ? s.x : 0.0), j == 0 ? s.y : 0.0);
    double ahead[kAhead];               // row k + 1 of H at columns threadIdx.x + q kSolveT
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
        const int j = threadIdx.x + q * kSolveT;
        ahead[q] = n > 1 && j < n ? Hr[(int64_t)n + j] : 0.0;
    }
    double bk = n > 1 ? Hr[n] : 0.0;
    __syncthreads();
    int64_t roff = 0;                   // offset of packed row k of R
    for (int k = 0; k + 1 < n; ++k) {
        const double *h = Hr + (int64_t)(k + 1) * n;   // row k + 1 (columns k.. are its nonzeros)
        double c;
        double2 sn;
        rotation(carry[k], bk, c, sn);
        const bool more = k + 2 < n;
        const double bnext = more ? h[n + k + 1] : 0.0;
        auto turn = [&](int j, double hj) {
            // R row k = c carry + sn next ; new carry = -conj(sn) carry + c next   (columns j >= k)
            const double2 a = carry[j];
            const double2 nx = make_double2(hj + (j == k + 1 ? s.x : 0.0), j == k + 1 ? s.y : 0.0);
            R[roff + (j - k)] = make_double2(c * a.x + (sn.x * nx.x - sn.y * nx.y), c * a.y + (sn.x * nx.y + sn.y * nx.x));
            if (j > k)
                carry[j] = make_double2(c * nx.x - (sn.x * a.x + sn.y * a.y), c * nx.y - (sn.x * a.y - sn.y * a.x));
        };
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int j = threadIdx.x + q * kSolveT;
            const double hj = ahead[q];
            if (more && j < n && j > k) ahead[q] = h[n + j];
            if (j >= k && j < n) turn(j, hj);
        }
        for (int j = threadIdx.x + kAhead * kSolveT; j < n; j += kSolveT)
            if (j >= k) turn(j, h[j]);
        // the same rotation on every right-hand side
        if ((int)threadIdx.x < cols) {
            double2 *yc = y + (int64_t)threadIdx.x * n;
            const double2 a = yc[k], b2 = yc[k + 1];
            yc[k] = make_double2(c * a.x + (sn.x * b2.x - sn.y * b2.y), c * a.y + (sn.x * b2.y + sn.y * b2.x));
            yc[k + 1] = make_double2(c * b2.x - (sn.x * a.x + sn.y * a.y), c * b2.y - (sn.x * a.y - sn.y * a.x));
        }
        bk = bnext;
        __syncthreads();
        roff += n - k;
    }
    if (threadIdx.x == 0) R[roff] = carry[n - 1];
    __syncthreads();
    // back substitution R x = y (rows packed: row i starts at i n - i (i - 1) / 2)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto row_of = [&](int i) { return (int64_t)i * n - (int64_t)i * (i - 1) / 2 - i; };   // + column
    for (int b0 = (n - 1) / 32 * 32; b0 >= 0; b0 -= 32) {
        const int nb = min(32, n - b0);
        for (int e = threadIdx.x; e < 32 * 32; e += kSolveT) {
            const int r = e / 32, c = e % 32;
            tri[c][r] = r < nb && c < nb && r <= c ? R[row_of(b0 + r) + b0 + c] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        for (int c = warp; c < cols; c += kSolveT / 32) {
            double2 *yc = y + (int64_t)c * n + b0;
            double2 v = lane < nb ? yc[lane] : make_double2(0.0, 0.0);
            const double2 d = lane < nb ? tri[lane][lane] : make_double2(1.0, 0.0);
            const double m = d.x * d.x + d.y * d.y;
            if (m == 0.0) atomicExch(singular, 1);
            const double2 di = m == 0.0 ? make_double2(0.0, 0.0) : make_double2(d.x / m, -d.y / m);
            for (int i = nb - 1; i >= 0; --i) {
                double2 xi = cmul(v, di);
                xi.x = __shfl_sync(0xffffffffu, xi.x, i);
                xi.y = __shfl_sync(0xffffffffu, xi.y, i);
                if (lane == i) v = xi;
                if (lane < i) {
                    const double2 p = cmul(tri[i][lane], xi);
                    v.x -= p.x;
                    v.y -= p.y;
                }
            }
            if (lane < nb) yc[lane] = v;
        }
        __syncthreads();
        // rows above: y_r -= sum over the block's columns, a warp per row
        for (int r = warp; r < b0; r += kSolveT / 32) {
            const double2 rv = lane < nb ? R[row_of(r) + b0 + lane] : make_double2(0.0, 0.0);
            for (int c = 0; c < cols; ++c) {
                double2 p = lane < nb ? cmul(rv, y[(int64_t)c * n + b0 + lane]) : make_double2(0.0, 0.0);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    p.x += __shfl_xor_sync(0xffffffffu, p.x, o);
                    p.y += __shfl_xor_sync(0xffffffffu, p.y, o);
                }
                if (lane == 0) {
                    y[(int64_t)c * n + r].x -= p.x;
                    y[(int64_t)c * n + r].y -= p.y;
                }
            }
        }
        __syncthreads();
    }
    for (int c = 0; c < cols; ++c)
        for (int i = threadIdx.x; i < n; i += kSolveT) {
            Cb[(int64_t)c * 2 * n + i] = y[(int64_t)c * n + i].x;
            Cb[(int64_t)c * 2 * n + n + i] = y[(int64_t)c * n + i].y;
        }
}

}  // namespace

bool hessenberg_applies(const plx_geom *g, int cols) {
    if (!g->has_T || g->n_var < 3) return false;
    // carry row and right-hand sides in one block's shared memory
    if ((size_t)(1 + cols) * g->n_var * sizeof(double2) > 200 * 1024) return false;
    if (g->model == PLX_BEM_DPCM) return true;
    return g->model == PLX_WFQ && g->n_types == 1;
}

// Shift s(w) of every frequency: A(w) = A0 + s(w) I.
static std::vector<Cplx> hessenberg_shifts(const plx_geom *g) {
    std::vector<Cplx> s(g->n_freq);
    for (int f = 0; f < g->n_freq; ++f) {
        if (is_bem(g)) {
            s[f] = g->bem_z[f];
        } else {
            // the charge diagonal -z(w) of the one atom type (upload_frequency_tables)
            const double w = g->omega[f], tau = g->tau[0], dn = g->density[0];
            const double den = 2.0 * dn * tau;
            s[f] = {-(w * (-w * tau) / den), -(w * (-1.0) / den)};
        }
    }
    return s;
}

void build_hessenberg(plx_geom *g) {
    if (g->d_hess_rows.p) return;
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int n = g->n_var;
    const HessTiles t = hess_tiles(n);
    DevArray<double> A, Q, vbuf, beta, sub, npart, yp, zp, sp;
    A.alloc(ctx, (size_t)n * n);
    Q.alloc(ctx, (size_t)n * n);
    vbuf.alloc(ctx, n);
    beta.alloc(ctx, 1);
    sub.alloc(ctx, n);
    npart.alloc(ctx, 2 * (size_t)t.nrc);
    yp.alloc(ctx, (size_t)t.ncc * 2 * n);
    zp.alloc(ctx, (size_t)t.nrc * n);
    sp.alloc(ctx, (size_t)t.nrc * t.ncc);
    if (is_bem(g)) {
        // D stored transposed (d_T[j][i] = D(i, j)) is D column-major
        PLX_CHECK_CUDA(cudaMemcpyAsync(A.p, g->d_T.p, (size_t)n * n * 8, cudaMemcpyDeviceToDevice, st));
    } else {
        wfq_a0<<<dim3(n, n_blocks(n, kT)), kT, 0, st>>>(n, g->d_rowptr.p, g->d_col.p, g->d_kval.p, g->d_T.p, A.p);
        ctx->launches++;
    }
    hess_identity<<<dim3(n_blocks(n, kT), n), kT, 0, st>>>(n, Q.p);
    hh_norm0<<<t.nrc, kT, 0, st>>>(t, A.p, npart.p);
    ctx->launches += 2;
    const size_t sm_gemv = (size_t)(t.rt + 3 * t.ct) * 8, sm_upd = (size_t)(6 * t.rt + 10 * t.ct) * 8;
    for (int k = 0; k + 2 < n; ++k) {
        const int c0 = (k + 1) / t.ct;                        // first column tile with columns right of k
        const dim3 grid(t.ncc - c0, t.nrc);
        double *np0 = npart.p + (k & 1) * t.nrc, *np1 = npart.p + ((k + 1) & 1) * t.nrc;
        launch_pdl(hh_gemv, grid, kT, sm_gemv, st, t, k, c0, A.p, Q.p, np0, vbuf.p, beta.p, sub.p, yp.p, zp.p, sp.p);
        launch_pdl(hh_update, grid, kT, sm_upd, st, t, k, c0, A.p, Q.p, vbuf.p, beta.p, yp.p, zp.p, sp.p, np1);
        ctx->launches += 2;
    }
    hess_rows<<<dim3(n_blocks(n, 32), n_blocks(n, 32)), dim3(32, 8), 0, st>>>(n, A.p, sub.p);
    ctx->launches++;
    PLX_CHECK_CUDA(cudaGetLastError());
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));
    g->d_hess_qt.swap(Q);
    g->d_hess_rows.swap(A);
}

// Solves A(w_f) x = b for the frequencies of `freqs` (cols right-hand sides each,
// B and X [freqs.size() * cols][2][n], frequency-major).  Returns false when a
// frequency's triangular factor has a zero on its diagonal (singular A(w)), or
// when there is no room beside T for three n x n matrices (H, Q^T and one frequency's
// triangular factor): the caller then factors A(w) per frequency, which needs two and
// the LU's work space.
static bool shifted_solve(plx_geom *g, const std::vector<int32_t> &freqs, int cols, const double *B, double *X) {
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int n = g->n_var;
    const int F = (int)freqs.size();
    const size_t rbytes = (size_t)n * (n + 1) / 2 * sizeof(double2);
    auto room = [&] { return ctx->budget > ctx->in_use ? ctx->budget - ctx->in_use : 0; };
    // no reduction for a solve that has no room
    if (ctx->budget && room() < rbytes + (g->d_hess_rows.p ? 0 : 16 * (uint64_t)n * n)) return false;
    build_hessenberg(g);
    if (F == 0) return true;
    const std::vector<Cplx> shifts = hessenberg_shifts(g);
    DevArray<Cplx> d_shift;
    d_shift.alloc(ctx, shifts.size());
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_shift.p, shifts.data(), shifts.size() * sizeof(Cplx), cudaMemcpyHostToDevice, st));
    const size_t smem = (size_t)(1 + cols) * n * sizeof(double2);
    if (smem > 200 * 1024) throw Error(PLX_ERR_UNSUPPORTED, "order too large for the shifted Hessenberg solve");
    once_per_device(reinterpret_cast<const void *>(hess_solve), ctx->device, [] {
        PLX_CHECK_CUDA(cudaFuncSetAttribute(hess_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    });
    // waves of frequencies whose triangular factors fit a quarter of the budget
    const int wave = (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)F, room() / 4 / rbytes));
    DevArray<double2> R;
    DevArray<int32_t> d_f;
    DevArray<int> sing;
    R.alloc(ctx, (size_t)wave * n * (n + 1) / 2);
    d_f.alloc(ctx, F);
    sing.alloc(ctx, 1);
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_f.p, freqs.data(), F * 4, cudaMemcpyHostToDevice, st));
    PLX_CHECK_CUDA(cudaMemsetAsync(sing.p, 0, sizeof(int), st));
    // a wave's Q^T b and x = Q y are one product each, in X and with the triangular
    // factors' memory for the partial sums (a product of the whole grid with memory of its
    // own took 167 MB at 893 unknowns and 61 frequencies)
    double *part = reinterpret_cast<double *>(R.p);
    const size_t prows = (size_t)wave * n * (n + 1);
    for (int f0 = 0; f0 < F; f0 += wave) {
        const int nf = std::min(wave, F - f0);
        double *x = X + (size_t)f0 * cols * 2 * n;
        product_in_room(ctx, part, prows, 2 * nf * cols, n, B + (size_t)f0 * cols * 2 * n, g->d_hess_qt.p, true, x);
        hess_solve<<<nf, kSolveT, smem, st>>>(n, cols, d_f.p + f0, d_shift.p, g->d_hess_rows.p, x, R.p, sing.p);
        ctx->launches++;
        PLX_CHECK_CUDA(cudaGetLastError());
        product_in_room(ctx, part, prows, 2 * nf * cols, n, x, g->d_hess_qt.p, false, x);
    }
    int hs = 0;
    PLX_CHECK_CUDA(cudaMemcpyAsync(&hs, sing.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));
    return hs == 0;
}

bool hessenberg_solve(plx_geom *g, const std::vector<int32_t> &freqs, int cols, const double *B, double *X) {
    try {
        return shifted_solve(g, freqs, cols, B, X);
    } catch (const Error &e) {
        if (e.code != PLX_ERR_BUDGET && e.code != PLX_ERR_NOMEM) throw;
        g->d_hess_qt.release();              // the LU gets the reduction's room
        g->d_hess_rows.release();
        return false;
    }
}

}  // namespace plx
