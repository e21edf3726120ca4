// The frequency-dependent operator A(w) = blockdiag(Kop(w), I) T + D(w) and
// the right-hand sides, for batches of columns (one frequency per column).
//
// Reference: product_matrix_vector_{wfq,wfqfmu} (wfq_module.f90:321-348,
// wfqfmu_module.f90:584-626) = T x (product_q_block_x / product_mu_block_x,
// matrix_module.f90:727-1001), then the charge rows through (K - P) or
// 1/2 (K + H(w)) (update_y_q, matrix_module.f90:1011-1098), dipole rows copied
// (update_y_mu, :1107-1125), then new_gmres_diagonal_shift.
#include <algorithm>

#include "pair_tiles.cuh"
#include "pdl.cuh"
#include "plx_internal.h"
#include "skinny.cuh"
#include "warp_sums.cuh"

namespace plx {

namespace {

// ---------------------------------------------------------------------------
// S = T X generated on the fly (matrix-free), at most CB columns per launch:
// one or several warps per target atom, the lanes over the source atoms.
//
// FP64 bound: a near pair costs three erf and two exp (alloy pairs four and
// three), a distant one about 40 operations, each column 32 FMAs.  One thread
// per target atom walking every source (the first form of this kernel) ran 16
// CTAs for 1,961 atoms: 3,383 us for one column; with the sources spread over the
// lanes, the width table and the undamped distant tile 96 us.  700 atoms, 4
// columns: 1,213 -> 34.5 us.
//
// Each lane adds its sources in ascending order with explicit FMAs, the lanes are
// added by a fixed exchange tree and the warps of a target in order; the number
// of warps depends on the number of atoms alone, so a column's sums depend
// neither on the batch nor on CB.
// ---------------------------------------------------------------------------
constexpr int kOtfWarps = 8;
constexpr int kOtfFewCols = 4;              // columns up to which it is used; the tiled form above
constexpr int kOtfNoScratch = 16;           // columns up to which a product goes on without the tiled form's scratch

// Warps per target atom: enough of them for ~24 warps on every SM of a B200 (148).  The
// split fixes the order of a target's sum, so it takes a constant, not the device's
// number of SMs: a solve gives the same bits on every device.
int otf_warps(int N) {
    int w = 1;
    while (w < kOtfWarps && (int64_t)N * w < 148 * 24) w *= 2;
    return w;
}

template <int CB, bool FMU>
__global__ void __launch_bounds__(32 * kOtfWarps) otf_contract(int N, int wt, int count, int nv, int nt,
                                                               const double *__restrict__ pos,
                                                               const double *__restrict__ par,
                                                               const int32_t *__restrict__ type,
                                                               const PairWidths *__restrict__ widths,
                                                               const double *__restrict__ X, double *__restrict__ S) {
    pdl_sync();
    constexpr int NC = FMU ? 4 : 1;            // components per atom
    constexpr int V = NC * 2 * CB;             // values per target: [component][part][column]
    __shared__ double red[kOtfWarps][V];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * (kOtfWarps / wt) + warp / wt, part = warp % wt;
    double acc[V];
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = 0.0;
    if (i < N) {
        const double xi = pos[i], yi = pos[N + i], zi = pos[2 * N + i];
        const int ti = type[i];
        for (int j = part * 32 + lane; j < N; j += 32 * wt) {
            double xq[2 * CB];
#pragma unroll
            for (int k = 0; k < 2 * CB; ++k) xq[k] = (k >> 1) < count ? X[(int64_t)k * nv + j] : 0.0;
            if (j == i) {
                const double eta = par[2 * N + i];
#pragma unroll
                for (int k = 0; k < 2 * CB; ++k) acc[k] = fma(eta, xq[k], acc[k]);
                continue;
            }
            const double dx = xi - pos[j], dy = yi - pos[N + j], dz = zi - pos[2 * N + j];
            const int tj = type[j];
            if (!FMU) {
                const double q = plx_pair_qq_w(dx, dy, dz, widths[ti + nt * tj]);
#pragma unroll
                for (int k = 0; k < 2 * CB; ++k) acc[k] = fma(q, xq[k], acc[k]);
                continue;
            }
            PairTile tl;
            plx_pair_tile_w(dx, dy, dz, widths[ti + nt * tj], ti == tj, tl);
#pragma unroll
            for (int k = 0; k < 2 * CB; ++k) {
                const double *xm = X + (int64_t)k * nv + N + 3LL * j;
                const bool in = (k >> 1) < count;
                const double m0 = in ? xm[0] : 0.0, m1 = in ? xm[1] : 0.0, m2 = in ? xm[2] : 0.0;
                acc[k] = fma(tl.qm[2], m2, fma(tl.qm[1], m1, fma(tl.qm[0], m0, fma(tl.qq, xq[k], acc[k]))));
                constexpr int P = 2 * CB;
                if (NC > 1) {
                    acc[P % V + k] = fma(tl.mm[2], m2, fma(tl.mm[1], m1, fma(tl.mm[0], m0,
                                         fma(tl.mq[0], xq[k], acc[P % V + k]))));
                    acc[2 * P % V + k] = fma(tl.mm[4], m2, fma(tl.mm[3], m1, fma(tl.mm[1], m0,
                                             fma(tl.mq[1], xq[k], acc[2 * P % V + k]))));
                    acc[3 * P % V + k] = fma(tl.mm[5], m2, fma(tl.mm[4], m1, fma(tl.mm[2], m0,
                                             fma(tl.mq[2], xq[k], acc[3 * P % V + k]))));
                }
            }
        }
    }
    const int base = lane_sums<V>(acc, lane);
    constexpr int L = V > 32 ? V / 32 : 1;      // sums a lane owns
    constexpr int G = V < 32 ? 32 / V : 1;      // lanes that own the same sum
    if (lane % G == 0) {
#pragma unroll
        for (int k = 0; k < L; ++k) red[warp][base + k] = acc[k];
    }
    __syncthreads();
    if (i >= N || part != 0) return;
    for (int e = lane; e < V; e += 32) {
        double s = red[warp][e];
        for (int w = 1; w < wt; ++w) s += red[warp + w][e];
        const int comp = e / (2 * CB), k = e % (2 * CB);
        if ((k >> 1) < count) S[(int64_t)k * nv + (comp == 0 ? i : N + 3 * i + comp - 1)] = s;
    }
}

// ---------------------------------------------------------------------------
// The same for many columns: S^T = X^T T with T generated in shared memory 16
// unknowns at a time, split over source atoms and reduced by skinny_reduce.  Rows
// and columns run atom by atom (an atom's charge, then its three dipole
// components), so a thread evaluates one pair of atoms and writes its 4 x 4
// block: the slab's erf and exp are evaluated once per pair instead of once per
// element.  BM rows of X^T a block (16, 32, 48 or 64): the fewest that hold the
// batch, so that 42 rows do not run as 64.  The products are FP64 matrix
// instructions, each of the four warps 32 columns.  Every kFlush slabs (256 unknowns)
// the sums move to a second set in shared memory: chains of thousands of terms cost
// accuracy (a smooth vector on 23,400 unknowns: 6.3e-15 of the norm in one chain a
// chunk, 4.4e-15 in the thread-per-atom form, now 0.7e-15).  The order of an element's
// sum does not depend on BM.
// Measured at 13,528 unknowns and 42 rows: 5,085 us element by element in 64 rows,
// 1,429 us a pair at a time with FMAs, now 1,083 us (average of four launches).
// ---------------------------------------------------------------------------
constexpr int BN = 128, kTiledThreads = 128;
constexpr int kFlush = 16;

template <int BM, bool FMU>
__global__ void __launch_bounds__(kTiledThreads) otf_tiled_partial(int R, int n, int jchunk, int N, int nt,
                                                                   const double *__restrict__ pos,
                                                                   const double *__restrict__ par,
                                                                   const int32_t *__restrict__ type,
                                                                   const PairWidths *__restrict__ widths,
                                                                   const double *__restrict__ Xt,
                                                                   double *__restrict__ part) {
    constexpr int NC = FMU ? 4 : 1;
    constexpr int KA = 16 / NC;                // source atoms a slab (16 unknowns)
    constexpr int CA = BN / NC;                // target atoms a block
    constexpr int MT = BM / 8, NT = BN / 32;   // 8 x 8 tiles of a warp
    __shared__ double As[BM][16 + 4];          // the paddings spread a fragment over the banks
    __shared__ __align__(16) double Bs[16][BN + 4];        // written two elements at a time
    static_assert((BN + 4) % 2 == 0 && BN % 4 == 0, "a row of Bs and an atom's components start at 16 bytes");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kk = lane & 3, g = lane >> 2;
    const int row0 = blockIdx.y * BM, i0 = blockIdx.x * CA;
    const int jbeg = blockIdx.z * jchunk, jend = min(N, jbeg + jchunk);
    double acc[MT][NT][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
    extern __shared__ double upper[];          // [MT * NT * 2][threads]: the second set
    for (int e = 0; e < MT * NT * 2; ++e) upper[e * kTiledThreads + threadIdx.x] = 0.0;
    auto flush = [&]() {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int t = 0; t < NT; ++t)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    upper[((m * NT + t) * 2 + v) * kTiledThreads + threadIdx.x] += acc[m][t][v];
                    acc[m][t][v] = 0.0;
                }
    };
    int slab = 0;
    for (int j0 = jbeg; j0 < jend; j0 += KA) {
        __syncthreads();
        for (int e = threadIdx.x; e < BM * 16; e += kTiledThreads) {
            const int r = e / 16, k = e % 16, gr = row0 + r, j = j0 + k / NC, comp = k % NC;
            As[r][k] = (gr < R && j < jend) ? Xt[(int64_t)gr * n + (comp == 0 ? j : N + 3 * j + comp - 1)] : 0.0;
        }
#pragma unroll 1
        for (int e = threadIdx.x; e < KA * CA; e += kTiledThreads) {
            const int jl = e / CA, il = e % CA, i = i0 + il, j = j0 + jl;
            if (!FMU) {
                double q = 0.0;
                if (i < N && j < jend)
                    q = i == j ? par[2 * N + i]
                               : plx_pair_qq_w(pos[i] - pos[j], pos[N + i] - pos[N + j], pos[2 * N + i] - pos[2 * N + j],
                                               widths[type[i] + nt * type[j]]);
                Bs[jl][il] = q;
                continue;
            }
            PairTile t;
            t.qq = 0.0;
#pragma unroll
            for (int k = 0; k < 3; ++k) t.qm[k] = t.mq[k] = 0.0;
#pragma unroll
            for (int k = 0; k < 6; ++k) t.mm[k] = 0.0;
            if (i < N && j < jend) {
                if (i == j) {
                    t.qq = par[2 * N + i];
                } else {
                    const int ti = type[i], tj = type[j];
                    plx_pair_tile_w(pos[i] - pos[j], pos[N + i] - pos[N + j], pos[2 * N + i] - pos[2 * N + j],
                                    widths[ti + nt * tj], ti == tj, t);
                }
            }
            // element [source component][target component]
            double2 *b = reinterpret_cast<double2 *>(&Bs[(NC * jl) % 16][(NC * il) % BN]);
            constexpr int ld = (BN + 4) / 2;
            b[0] = make_double2(t.qq, t.mq[0]);
            b[1] = make_double2(t.mq[1], t.mq[2]);
            b[ld] = make_double2(t.qm[0], t.mm[0]);
            b[ld + 1] = make_double2(t.mm[1], t.mm[2]);
            b[2 * ld] = make_double2(t.qm[1], t.mm[1]);
            b[2 * ld + 1] = make_double2(t.mm[3], t.mm[4]);
            b[3 * ld] = make_double2(t.qm[2], t.mm[2]);
            b[3 * ld + 1] = make_double2(t.mm[4], t.mm[5]);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; k += 4) {      // unknowns past the chunk are zeros
            double a[MT], b[NT];
#pragma unroll
            for (int m = 0; m < MT; ++m) a[m] = As[8 * m + g][k + kk];
#pragma unroll
            for (int t = 0; t < NT; ++t) b[t] = Bs[k + kk][32 * warp + 8 * t + g];
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int t = 0; t < NT; ++t) dmma(acc[m][t], a[m], b[t]);
        }
        if (++slab % kFlush == 0) flush();
    }
    flush();
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const int gr = row0 + 8 * m + g;
        if (gr >= R) continue;
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int c = 32 * warp + 8 * t + 2 * kk + v, i = i0 + c / NC, comp = c % NC;
                if (i < N)
                    part[((int64_t)blockIdx.z * R + gr) * n + (comp == 0 ? i : N + 3 * i + comp - 1)] =
                        upper[((m * NT + t) * 2 + v) * kTiledThreads + threadIdx.x];
            }
    }
}

// ---------------------------------------------------------------------------
// Charge rows: y_i = sum_j c_ij (s_j - s_i), c_ij = K_ij (one atom type) or
// 1/2 (K_ij + (w_tj/w_ti) K_ji) (several types), then + D_q(w) x_i.
// One warp per row and a chunk of kChargeCols columns.  A row of K holds a few
// hundred entries (the Fermi damping reaches ~4 nearest-neighbour distances);
// each lane keeps its share of the row (entries lane, lane + 32, ...) in
// registers and reuses it for every column, so the CSR is read once per row
// and chunk instead of once per column.  Per column every lane sums its
// entries in CSR order and the warp adds the lanes with a fixed butterfly, so
// a column's result does not depend on the batch it is in.
// ---------------------------------------------------------------------------
constexpr int kChargeCols = 32;
constexpr int kChargeReg = 16;              // entries per lane held in registers (rows up to 512)

template <bool HETERO>
__device__ __forceinline__ void charge_term(int nt, int ti, int tj, int f, double k, double kt,
                                            const Cplx *__restrict__ wratio, double dre, double dim,
                                            double &yre, double &yim) {
    if (!HETERO) {
        yre = fma(k, dre, yre);
        yim = fma(k, dim, yim);
    } else {
        Cplx w = wratio[ti + nt * tj + (int64_t)nt * nt * f];
        double cre = 0.5 * (k + w.re * kt), cim = 0.5 * (w.im * kt);
        yre += cre * dre - cim * dim;
        yim += cre * dim + cim * dre;
    }
}

// y (times sign) + D_q(w) x of one row and column
__device__ __forceinline__ void charge_store(int nv, int c, int i, const Cplx &d, const double *__restrict__ X,
                                             double *__restrict__ Y, double sign, int add_diag, double yre, double yim) {
    yre *= sign;
    yim *= sign;
    if (add_diag) {
        const double xr = X[(int64_t)c * 2 * nv + i], xi = X[(int64_t)c * 2 * nv + nv + i];
        yre += d.re * xr - d.im * xi;
        yim += d.re * xi + d.im * xr;
    }
    Y[(int64_t)c * 2 * nv + i] = yre;
    Y[(int64_t)c * 2 * nv + nv + i] = yim;
}

template <bool HETERO>
__global__ void __launch_bounds__(256) charge_rows(int N, int nt, int nv, int count,
                                                   const int32_t *__restrict__ freq,
                                                   const int32_t *__restrict__ type,
                                                   const int32_t *__restrict__ rowptr,
                                                   const int32_t *__restrict__ col,
                                                   const double *__restrict__ kval,
                                                   const double *__restrict__ ktval,
                                                   const Cplx *__restrict__ wratio, const Cplx *__restrict__ dq,
                                                   const double *__restrict__ S, const double *__restrict__ X,
                                                   double *__restrict__ Y, double sign, int add_diag) {
    pdl_sync();
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= N) return;
    const int c0 = blockIdx.y * kChargeCols;
    const int c1 = min(count, c0 + kChargeCols);
    const int e0 = rowptr[i], e1 = rowptr[i + 1];
    const bool in_reg = e1 - e0 <= 32 * kChargeReg;
    const int ti = type[i];
    constexpr int HR = HETERO ? kChargeReg : 1;
    int rj[kChargeReg], rt[HR];
    double rk[kChargeReg], rkt[HR];
#pragma unroll
    for (int t = 0; t < kChargeReg; ++t) {
        const int e = e0 + lane + 32 * t;
        const bool live = in_reg && e < e1;
        rj[t] = live ? col[e] : 0;
        rk[t] = live ? kval[e] : 0.0;
        if (HETERO) {
            rkt[t % HR] = live ? ktval[e] : 0.0;
            rt[t % HR] = live ? type[rj[t]] : 0;
        }
    }
    for (int c = c0; c < c1; ++c) {
        const int f = freq[c];
        const double *sr = S + (int64_t)c * 2 * nv;
        const double *si = sr + nv;
        const double s_re = sr[i], s_im = si[i];
        double yre = 0.0, yim = 0.0;
        if (in_reg) {
#pragma unroll
            for (int t = 0; t < kChargeReg; ++t) {
                if (e0 + lane + 32 * t < e1) {
                    const int j = rj[t];
                    charge_term<HETERO>(nt, ti, HETERO ? rt[t % HR] : 0, f, rk[t], HETERO ? rkt[t % HR] : 0.0,
                                        wratio, sr[j] - s_re, si[j] - s_im, yre, yim);
                }
            }
        } else {
            for (int e = e0 + lane; e < e1; e += 32) {
                const int j = col[e];
                charge_term<HETERO>(nt, ti, HETERO ? type[j] : 0, f, kval[e], HETERO ? ktval[e] : 0.0, wratio,
                                    sr[j] - s_re, si[j] - s_im, yre, yim);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            yre += __shfl_xor_sync(0xffffffffu, yre, o);
            yim += __shfl_xor_sync(0xffffffffu, yim, o);
        }
        if (lane == 0) charge_store(nv, c, i, dq[ti + nt * f], X, Y, sign, add_diag, yre, yim);
    }
}

// The same rows of one atom type for many columns, with columns across the lanes.
// The row form gathers S at the row's atoms, a cache line per entry and column: at 893
// sodium atoms (289 entries a row) x 61 columns it was bound by L1, 78 us.  Here S is
// transposed first (St[atom][column], 16 bytes a column), so that an entry is one
// coalesced read of 32 columns: 28 us with the transpose, bound by instruction issue
// (a shuffle for the entry's place and two for its coefficient).  Four warps share a row
// and 32 columns: warp m sums the entries of the row form's lanes m, m + 4, ..., eight
// chains a thread, each in CSR order, and the chains are added in the butterfly's order
// -- every result has the row form's bits.
//
// From 12 columns: the transposed form takes the same time for 1 to 32, the row form
// grows with them (893 atoms, 8 / 12 / 32 columns: 18.5 / 25 / 70 us against 14 / 15 /
// 16; 1,961 silver atoms: 25 / 36 / 90 against 30 / 31 / 32; 4,693 sodium atoms:
// 49 / 72 / 183 against 67 / 69 / 72).
constexpr int kColsMin = 12;
__global__ void __launch_bounds__(128, 7) charge_cols(
    int N, int nt, int nv, int count, const int32_t *__restrict__ freq, const int32_t *__restrict__ type,
    const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col, const double *__restrict__ kval,
    const Cplx *__restrict__ dq, const double2 *__restrict__ St, const double *__restrict__ X, double *__restrict__ Y,
    double sign, int add_diag) {
    pdl_sync();
    __shared__ double2 part[4][32];
    const int i = blockIdx.x, lane = threadIdx.x & 31, m = threadIdx.x >> 5;
    const int c = blockIdx.y * 32 + lane;
    const double2 *col_s = St + min(c, count - 1);
    const double2 s = col_s[(int64_t)i * count];
    const int e1 = rowptr[i + 1];
    double yre[8], yim[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) yre[q] = yim[q] = 0.0;
    // lane l (l mod 8) holds the warp's entry 4 l + m of the 32 in turn
    int e = rowptr[i] + m + 4 * (lane & 7);
    int at = 0;
    double k = 0.0;
    auto fetch = [&] {
        at = (e < e1 ? col[e] : 0) * count;
        k = e < e1 ? kval[e] : 0.0;
    };
    fetch();
    int left = e1 - rowptr[i];
    for (; left >= 32; left -= 32) {
        double2 v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = col_s[__shfl_sync(0xffffffffu, at, q)];
        const double kk = k;
        e += 32;
        fetch();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double kq = __shfl_sync(0xffffffffu, kk, q);
            yre[q] = fma(kq, v[q].x - s.x, yre[q]);
            yim[q] = fma(kq, v[q].y - s.y, yim[q]);
        }
    }
    {
        double2 v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = col_s[__shfl_sync(0xffffffffu, at, q)];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const double kq = __shfl_sync(0xffffffffu, k, q);
            if (4 * q + m < left) {
                yre[q] = fma(kq, v[q].x - s.x, yre[q]);
                yim[q] = fma(kq, v[q].y - s.y, yim[q]);
            }
        }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < o; ++q) {
            yre[q] += yre[q + o];
            yim[q] += yim[q + o];
        }
    part[m][lane] = make_double2(yre[0], yim[0]);
    __syncthreads();
    if (m != 0 || c >= count) return;
    const double2 p0 = part[0][lane], p1 = part[1][lane], p2 = part[2][lane], p3 = part[3][lane];
    charge_store(nv, c, i, dq[type[i] + nt * freq[c]], X, Y, sign, add_diag, (p0.x + p2.x) + (p1.x + p3.x),
                 (p0.y + p2.y) + (p1.y + p3.y));
}

// St[i][r] = S[r][i] for the charges i < N of R rows of length nv.
__global__ void __launch_bounds__(256) transpose_charges(int N, int nv, int R, const double *__restrict__ S,
                                                         double *__restrict__ St) {
    pdl_sync();
    __shared__ double tile[32][33];
    const int i0 = blockIdx.x * 32, r0 = blockIdx.y * 32, x = threadIdx.x & 31, y = threadIdx.x >> 5;
#pragma unroll
    for (int q = y; q < 32; q += 8)
        if (r0 + q < R && i0 + x < N) tile[q][x] = S[(int64_t)(r0 + q) * nv + i0 + x];
    __syncthreads();
#pragma unroll
    for (int q = y; q < 32; q += 8)
        if (i0 + q < N && r0 + x < R) St[(int64_t)(i0 + q) * R + r0 + x] = tile[x][q];
}

// Dipole rows: y = s + (sum_t f_t,i / alpha_t(w)) x.
__global__ void dipole_rows(int N, int nt, int nv, int count, const int32_t *__restrict__ freq,
                            const double *__restrict__ frac, const Cplx *__restrict__ inv_alpha,
                            const double *__restrict__ S, const double *__restrict__ X,
                            double *__restrict__ Y) {
    pdl_sync();
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int c = blockIdx.y;
    if (e >= 3LL * N || c >= count) return;
    int i = (int)(e / 3);
    int f = freq[c];
    double zre = 0.0, zim = 0.0;
    for (int t = 0; t < nt; ++t) {
        double fr = frac[t + (int64_t)nt * i];
        Cplx a = inv_alpha[t + nt * f];
        zre += fr * a.re;
        zim += fr * a.im;
    }
    int64_t r = N + e;
    const double *sc = S + (int64_t)c * 2 * nv;
    const double *xc = X + (int64_t)c * 2 * nv;
    double xr = xc[r], xi = xc[nv + r];
    Y[(int64_t)c * 2 * nv + r] = sc[r] + zre * xr - zim * xi;
    Y[(int64_t)c * 2 * nv + nv + r] = sc[nv + r] + zre * xi + zim * xr;
}

// Alloy correction after the folded contraction: for every interface row i,
//   y_i += sum_{j of another type} 1/2 (w_tj/w_ti(w) - 1) K_ji (s_j - s_i),
// s = T x of the interface atoms (rows n + position in J of the output).
// One thread per (interface row, column).
__global__ void iface_rows(int nx, int count, int nt, int nv, int64_t ldS, const int32_t *__restrict__ freq,
                           const int32_t *__restrict__ type, const int32_t *__restrict__ xrow,
                           const int32_t *__restrict__ xipos, const int32_t *__restrict__ xrowptr,
                           const int32_t *__restrict__ xcol, const int32_t *__restrict__ xtj,
                           const double *__restrict__ xkt, const Cplx *__restrict__ wratio,
                           const double *__restrict__ S, double *__restrict__ Y) {
    pdl_sync();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = blockIdx.y;
    if (t >= nx || c >= count) return;
    const int i = xrow[t], f = freq[c], ti = type[i];
    const double *sr = S + (int64_t)c * 2 * ldS + nv, *si = sr + ldS;
    const double s_re = sr[xipos[t]], s_im = si[xipos[t]];
    double yre = 0.0, yim = 0.0;
    for (int e = xrowptr[t]; e < xrowptr[t + 1]; ++e) {
        const int p = xcol[e];
        const Cplx w = wratio[ti + nt * xtj[e] + (int64_t)nt * nt * f];
        const double cre = 0.5 * (w.re - 1.0) * xkt[e], cim = 0.5 * w.im * xkt[e];
        const double dre = sr[p] - s_re, dim = si[p] - s_im;
        yre += cre * dre - cim * dim;
        yim += cre * dim + cim * dre;
    }
    Y[(int64_t)c * 2 * nv + i] += yre;
    Y[(int64_t)c * 2 * nv + nv + i] += yim;
}

// Static potential V_i (field along pol) for the right-hand side.
__global__ void potential_kernel(int N, int nv, int count, const int32_t *__restrict__ pol,
                                 const double *__restrict__ pos, double e0, int use_min,
                                 double mx, double my, double mz, double *__restrict__ V) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int c = blockIdx.y;
    if (i >= nv || c >= count) return;
    double v = 0.0;
    if (i < N) {
        int p = pol[c];
        double x = pos[(int64_t)p * N + i];
        double m = p == 0 ? mx : (p == 1 ? my : mz);
        v = use_min ? -e0 * fabs(x - m) : -e0 * x;
    }
    V[(int64_t)c * 2 * nv + i] = v;
    V[(int64_t)c * 2 * nv + nv + i] = 0.0;
}

// Dipole part of the right-hand side: E0 on the polarisation component.
__global__ void rhs_dipole(int N, int nv, int count, const int32_t *__restrict__ pol, double e0,
                           double *__restrict__ B) {
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int c = blockIdx.y;
    if (e >= 3LL * N || c >= count) return;
    int k = (int)(e % 3);
    B[(int64_t)c * 2 * nv + N + e] = (k == pol[c]) ? e0 : 0.0;
    B[(int64_t)c * 2 * nv + nv + N + e] = 0.0;
}

// Frequency-independent parts of diag(blockdiag(Kop, I) T) on the charge rows.
__global__ void diag_parts(int N, int nt, const double *__restrict__ pos, const double *__restrict__ par,
                           const int32_t *__restrict__ type, const int32_t *__restrict__ rowptr,
                           const int32_t *__restrict__ col, const double *__restrict__ kval,
                           const double *__restrict__ ktval, double *__restrict__ a, double *__restrict__ b) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    double eta = par[2 * N + i], rq = par[i];
    double sa = 0.0;
    for (int t = 0; t < nt; ++t) b[(int64_t)i * nt + t] = 0.0;
    for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) {
        int j = col[e];
        double tij = plx_pair_qq(pos[i] - pos[j], pos[N + i] - pos[N + j], pos[2 * N + i] - pos[2 * N + j], rq,
                                 par[j]);
        sa += kval[e] * (tij - eta);
        b[(int64_t)i * nt + type[j]] += ktval[e] * (tij - eta);
    }
    a[i] = sa;
}

// 1 / diag(A(w)) per column.
__global__ void diag_inverse_kernel(int N, int nt, int nv, int count, int hetero, const int32_t *__restrict__ freq,
                                    const int32_t *__restrict__ type, const double *__restrict__ a,
                                    const double *__restrict__ b, const Cplx *__restrict__ wratio,
                                    const Cplx *__restrict__ dq, const double *__restrict__ frac,
                                    const Cplx *__restrict__ inv_alpha, double *__restrict__ P) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    int c = blockIdx.y;
    if (r >= nv || c >= count) return;
    int f = freq[c];
    double re, im;
    if (r < N) {
        int ti = type[r];
        if (!hetero) {
            re = a[r];
            im = 0.0;
        } else {
            re = a[r];
            im = 0.0;
            for (int t = 0; t < nt; ++t) {
                Cplx w = wratio[ti + nt * t + (int64_t)nt * nt * f];
                double bt = b[(int64_t)r * nt + t];
                re += w.re * bt;
                im += w.im * bt;
            }
            re *= 0.5;
            im *= 0.5;
        }
        Cplx d = dq[ti + nt * f];
        re += d.re;
        im += d.im;
    } else {
        int i = (r - N) / 3;
        re = 0.0;
        im = 0.0;
        for (int t = 0; t < nt; ++t) {
            double fr = frac[t + (int64_t)nt * i];
            Cplx al = inv_alpha[t + nt * f];
            re += fr * al.re;
            im += fr * al.im;
        }
    }
    double m = re * re + im * im;
    double *pc = P + (int64_t)c * 2 * nv;
    pc[r] = m > 0.0 ? re / m : 1.0;
    pc[nv + r] = m > 0.0 ? -im / m : 0.0;
}

}  // namespace

void diagonal_inverse(plx_geom *g, const OpBatch &b, double *Pinv) {
    if (is_bem(g)) {
        bem_diagonal_inverse(g, b, Pinv);
        return;
    }
    plx_ctx *ctx = g->ctx;
    const int N = g->n_atoms, nt = g->n_types;
    if (!g->d_diag_a.p) {
        DevArray<double> a, b_;              // the geometry's once both are there
        a.alloc(ctx, N);
        b_.alloc(ctx, (size_t)N * nt);
        diag_parts<<<n_blocks(N, 128), 128, 0, ctx->stream>>>(N, nt, g->d_pos.p, g->d_par.p, g->d_type.p,
                                                              g->d_rowptr.p, g->d_col.p, g->d_kval.p,
                                                              g->d_ktval.p, a.p, b_.p);
        ctx->launches++;
        g->d_diag_a.swap(a);
        g->d_diag_b.swap(b_);
    }
    diag_inverse_kernel<<<dim3(n_blocks(g->n_var, 256), b.count), 256, 0, ctx->stream>>>(
        N, nt, g->n_var, b.count, nt > 1, b.d_freq, g->d_type.p, g->d_diag_a.p, g->d_diag_b.p, g->d_wratio.p,
        g->d_dq.p, g->d_frac.p, g->d_inv_alpha.p, Pinv);
    ctx->launches++;
    PLX_CHECK_CUDA(cudaGetLastError());
}

void contract_t_impl(plx_geom *g, int count, const double *X, double *S, bool on_the_fly);

void prof_begin(plx_ctx *ctx) {
    if (!ctx->profile) return;
    if (ctx->prof_used + 2 > ctx->prof_events.size()) {
        for (int k = 0; k < 2; ++k) {
            cudaEvent_t e;
            PLX_CHECK_CUDA(cudaEventCreate(&e));
            ctx->prof_events.push_back(e);
        }
    }
    PLX_CHECK_CUDA(cudaEventRecord(ctx->prof_events[ctx->prof_used], ctx->stream));
}

void prof_end(plx_ctx *ctx, int cat, double flops, double bytes) {
    if (!ctx->profile) return;
    PLX_CHECK_CUDA(cudaEventRecord(ctx->prof_events[ctx->prof_used + 1], ctx->stream));
    if (ctx->prof_cat.size() < ctx->prof_events.size() / 2) ctx->prof_cat.resize(ctx->prof_events.size() / 2);
    ctx->prof_cat[ctx->prof_used / 2] = cat;
    ctx->prof_used += 2;
    ctx->prof_flops[cat] += flops;
    ctx->prof_bytes[cat] += bytes;
    ctx->prof_launches[cat] += 1;
}

void contract_t(plx_geom *g, int count, const double *X, double *S, Contraction how) {
    plx_ctx *ctx = g->ctx;
    const double nn = (double)g->n_var;
    const bool otf = how == Contraction::FP64_OTF;
    if (otf && is_bem(g))
        throw Error(PLX_ERR_UNSUPPORTED, "BEM on the fly is not provided (the reference's BEM has no "
                                         "on-the-fly product either); use the on-memory mode");
    prof_begin(ctx);
    // algorithmic: 2 n^2 flops per real column (one product, whatever the
    // emulation); bytes: the stored T once at its storage precision, plus the
    // columns in and out
    double tbytes = 0.0;
    if (how == Contraction::TC3 || how == Contraction::TC1) {
        tc_contract(g, count, X, S, how == Contraction::TC3 ? 3 : 1);
        tbytes = (how == Contraction::TC3 ? 4.0 : 2.0) * nn * (double)g->ldk;
    } else {
        contract_t_impl(g, count, X, S, otf);
        tbytes = otf ? 0.0 : 8.0 * nn * nn;
    }
    prof_end(ctx, (how == Contraction::TC3 || how == Contraction::TC1) ? PROF_TC : PROF_FP64,
             2.0 * nn * nn * 2.0 * count, tbytes + 2.0 * 8.0 * nn * 2.0 * count);
}

// S = X T for R rows X [R][n] and a row-major n x n FP64 matrix (S^T = T^T X^T):
// the split-K products of skinny.cuh, the partial sums in `scratch` (grown on demand).
// A row's result does not depend on R.
void stored_product(plx_ctx *ctx, DevArray<double> &scratch, int R, int n, const double *X, const double *T, double *S) {
    int ks, kchunk;
    skinny_split(n, ks, kchunk);
    const size_t need = (size_t)ks * R * n;
    if (scratch.n < need) scratch.alloc(ctx, need);
    product_in_room(ctx, scratch.p, need, R, n, X, T, false, S);
}

void product_in_room(plx_ctx *ctx, double *scratch, size_t room, int R, int n, const double *X, const double *T,
                     bool transposed, double *S) {
    // K split: depends on n only (not on the batch)
    int ks, kchunk;
    skinny_split(n, ks, kchunk);
    const int most = (int)std::min<size_t>((size_t)R, room / ((size_t)ks * n));
    if (most < 1) throw Error(PLX_ERR_ARG, "no room for a row of the product");
    cudaStream_t st = ctx->stream;
    for (int r0 = 0; r0 < R; r0 += most) {
        const int nr = std::min(most, R - r0);
        const int64_t at = (int64_t)r0 * n;
        if (transposed) launch_product_partial<true>(st, nr, n, ks, kchunk, X + at, T, scratch);
        else launch_product_partial(st, nr, n, ks, kchunk, X + at, T, scratch);
        launch_pdl(skinny_reduce, n_blocks((int64_t)nr * n, 256), 256, 0, st, n, nr, ks, scratch, S + at);
        ctx->launches += 2;
    }
    PLX_CHECK_CUDA(cudaGetLastError());
}

// Matrix-free product four columns at a time; needs no scratch.
static void otf_few_columns(plx_geom *g, int count, const double *X, double *S) {
    plx_ctx *ctx = g->ctx;
    const bool fmu = g->model == PLX_WFQFMU;
    const int n = g->n_var, N = g->n_atoms;
    const int wt = otf_warps(N), blocks = n_blocks(N, kOtfWarps / wt);
    for (int c0 = 0; c0 < count; c0 += kOtfFewCols) {
        const int cb = std::min(kOtfFewCols, count - c0);
        const int64_t at = (int64_t)c0 * 2 * n;
#define PLX_OTF(CB, F)                                                                                            \
    launch_pdl(otf_contract<CB, F>, blocks, 32 * kOtfWarps, 0, ctx->stream, N, wt, cb, n, g->n_types, g->d_pos.p,    \
               g->d_par.p, g->d_type.p, g->d_widths.p, X + at, S + at)
        if (fmu) {
            if (cb == 1) PLX_OTF(1, true);
            else if (cb == 2) PLX_OTF(2, true);
            else PLX_OTF(4, true);
        } else {
            if (cb == 1) PLX_OTF(1, false);
            else if (cb == 2) PLX_OTF(2, false);
            else PLX_OTF(4, false);
        }
#undef PLX_OTF
        ctx->launches++;
    }
    PLX_CHECK_CUDA(cudaGetLastError());
}

void contract_t_impl(plx_geom *g, int count, const double *X, double *S, bool on_the_fly) {
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int n = g->n_var;
    const int R = 2 * count;
    if (on_the_fly) {
        const bool fmu = g->model == PLX_WFQFMU;
        const int N = g->n_atoms;
        if (count > kOtfFewCols) {
            // many columns: tiled product with T generated per slab; the split over the
            // sources depends on the number of atoms only (592: four blocks an SM of a B200;
            // constant for the same bits on every device)
            const int ca = fmu ? BN / 4 : BN, ka = fmu ? 4 : 16;
            const int tiles = n_blocks(N, ca);
            int js = std::max(1, std::min(64, (592 + tiles - 1) / tiles));
            const int jchunk = n_blocks(n_blocks(N, js), ka) * ka;
            js = n_blocks(N, jchunk);
            const size_t need = (size_t)js * R * n;
            if (g->d_part.n < need) {
                try {
                    g->d_part.alloc(ctx, need);
                } catch (const Error &) {
                    if (count > kOtfNoScratch) throw;
                    otf_few_columns(g, count, X, S);     // no room for the partial sums
                    return;
                }
            }
            // rows a block: all of them up to 64, or 16 as long as that gives no more than two
            // blocks an SM of a B200: a block's time is then its latency, and evaluating its
            // pairs again costs less than its rows (100 sodium atoms, 130 columns, with the sum:
            // 21.3 us in blocks of 64 rows, 17.6 in 16; element by element before: 17.8)
            const bool few = (int64_t)tiles * js * n_blocks(R, 16) <= 296;
            const int bm = few || R <= 16 ? 16 : R <= 32 ? 32 : (R <= 48 ? 48 : 64);
            const dim3 grid(tiles, n_blocks(R, bm), js);
#define PLX_OTF(BMV, F)                                                                                            \
    {                                                                                                             \
        auto kern = otf_tiled_partial<BMV, F>;                                                                    \
        const size_t smem = (size_t)BMV * BN * sizeof(double);                                                    \
        once_per_device(reinterpret_cast<const void *>(kern), ctx->device, [&] {                                  \
            PLX_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));   \
        });                                                                                                       \
        kern<<<grid, kTiledThreads, smem, st>>>(R, n, jchunk, N, g->n_types, g->d_pos.p, g->d_par.p, g->d_type.p, \
                                                g->d_widths.p, X, g->d_part.p);                                   \
    }
            if (fmu) {
                if (bm == 16) PLX_OTF(16, true)
                else if (bm == 32) PLX_OTF(32, true)
                else if (bm == 48) PLX_OTF(48, true)
                else PLX_OTF(64, true)
            } else {
                if (bm == 16) PLX_OTF(16, false)
                else if (bm == 32) PLX_OTF(32, false)
                else if (bm == 48) PLX_OTF(48, false)
                else PLX_OTF(64, false)
            }
#undef PLX_OTF
            launch_pdl(skinny_reduce, n_blocks((int64_t)R * n, 256), 256, 0, st, n, R, js, g->d_part.p, S);
            ctx->launches += 2;
            PLX_CHECK_CUDA(cudaGetLastError());
            return;
        }
        otf_few_columns(g, count, X, S);
        return;
    }
    if (!g->has_T) throw Error(PLX_ERR_ARG, "geometry was created without the dense T matrix");
    stored_product(ctx, g->d_part, R, n, X, g->d_T.p, S);
}

// Whether charge_cols takes a batch (its places are 32-bit).
static bool charges_by_column(const plx_geom *g, int count) {
    return g->n_types == 1 && count >= kColsMin && (int64_t)g->n_atoms * count <= INT32_MAX;
}

// The charge rows of a batch; St: room for the transposed S (2 count N doubles), or null.
static void charge_part(plx_geom *g, const OpBatch &b, const double *S, const double *X, double *Y, double sign,
                        int add_diag, double *St) {
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int N = g->n_atoms, nv = g->n_var;
    if (charges_by_column(g, b.count) && St) {
        const int R = 2 * b.count;
        launch_pdl(transpose_charges, dim3(n_blocks(N, 32), n_blocks(R, 32)), 256, 0, st, N, nv, R, S, St);
        launch_pdl(charge_cols, dim3(N, n_blocks(b.count, 32)), 128, 0, st, N, g->n_types, nv, b.count,
                   b.d_freq, g->d_type.p, g->d_rowptr.p, g->d_col.p, g->d_kval.p, g->d_dq.p,
                   reinterpret_cast<const double2 *>(St), X, Y, sign, add_diag);
        ctx->launches += 2;
        return;
    }
    const dim3 gq(n_blocks((int64_t)N * 32, 256), n_blocks(b.count, kChargeCols));
    launch_pdl(g->n_types > 1 ? charge_rows<true> : charge_rows<false>, gq, 256, 0, st, N, g->n_types, nv, b.count,
               b.d_freq, g->d_type.p, g->d_rowptr.p, g->d_col.p, g->d_kval.p, g->d_ktval.p, g->d_wratio.p, g->d_dq.p, S,
               X, Y, sign, add_diag);
    ctx->launches++;
}

static void finish_rows(plx_geom *g, const OpBatch &b, const double *S, const double *X,
                        double *Y) {
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int N = g->n_atoms, nv = g->n_var;
    // the product's partial sums have been added: their scratch holds the transpose
    charge_part(g, b, S, X, Y, 1.0, 1, g->d_part.n >= (size_t)b.count * 2 * N ? g->d_part.p : nullptr);
    if (g->model == PLX_WFQFMU) {
        dim3 gm(n_blocks(3LL * N, 256), b.count);
        launch_pdl(dipole_rows, gm, 256, 0, st, N, g->n_types, nv, b.count, b.d_freq, g->d_frac.p, g->d_inv_alpha.p, S,
                   X, Y);
        ctx->launches++;
    }
    PLX_CHECK_CUDA(cudaGetLastError());
}

// Output of the folded tensor-core contraction of b.count columns: the work
// array, or for alloys (interface rows after the n operator rows) the
// geometry's fold buffer.
static double *folded_output(plx_geom *g, const OpBatch &b, double *work) {
    const int64_t M = tc_fold_rows(g);
    if (M <= g->n_var) return work;
    const size_t need = (size_t)b.count * 2 * M;
    if (g->d_fold_work.n < need) g->d_fold_work.alloc(g->ctx, need);
    return g->d_fold_work.p;
}

// The interface correction of alloys after a folded contraction that has left
// Y = A0 X + D(w) X and the interface atoms' T x in S.
static void folded_finish(plx_geom *g, const OpBatch &b, const double *S, double *Y) {
    if (g->n_xrows == 0) return;
    plx_ctx *ctx = g->ctx;
    prof_begin(ctx);
    launch_pdl(iface_rows, dim3(n_blocks(g->n_xrows, 128), b.count), 128, 0, ctx->stream, g->n_xrows, b.count,
               g->n_types, g->n_var, g->fold_rows, b.d_freq, g->d_type.p, g->d_xrow.p, g->d_xipos.p, g->d_xrowptr.p,
               g->d_xcol.p, g->d_xtj.p, g->d_xkt.p, g->d_wratio.p, S, Y);
    ctx->launches++;
    PLX_CHECK_CUDA(cudaGetLastError());
    prof_end(ctx, PROF_ROWS, 0.0, 0.0);
}

static double tc_bytes(plx_geom *g, Contraction how, int count) {
    const double nn = (double)g->n_var;
    const double rows = tc_folds_operator(g) ? (double)g->fold_rows : nn;
    return (how == Contraction::TC3 ? 4.0 : 2.0) * rows * (double)g->ldk + 2.0 * 8.0 * nn * 2.0 * count;
}

// A tensor-core application: one contraction with the folded matrix (BEM: with D)
// whose output rows already carry the diagonal, Y = A0 X + D(w) X.
static TcItem tc_item(plx_geom *g, const OpBatch &b, const double *X, double *Y, double *work, Contraction how,
                      bool presplit) {
    const bool folds = tc_folds_operator(g);
    return TcItem{g,     b.count, X, folds ? folded_output(g, b, work) : work, how == Contraction::TC3 ? 3 : 1, folds,
                  b.d_freq, Y,    presplit};
}

void apply_operator(plx_geom *g, const OpBatch &b, const double *X, double *Y, double *work,
                    Contraction how, bool presplit) {
    if (b.count == 0) return;
    if (how == Contraction::TC3 || how == Contraction::TC1) {
        plx_ctx *ctx = g->ctx;
        const double nn = (double)g->n_var;
        const TcItem it = tc_item(g, b, X, Y, work, how, presplit);
        prof_begin(ctx);
        tc_contract_group({it});
        prof_end(ctx, PROF_TC, 2.0 * nn * nn * 2.0 * b.count, tc_bytes(g, how, b.count));
        if (it.folded) folded_finish(g, b, it.S, Y);
        return;
    }
    contract_t(g, b.count, X, work, how);
    prof_begin(g->ctx);
    if (is_bem(g))
        bem_apply_rows(g, b, work, X, Y);
    else
        finish_rows(g, b, work, X, Y);
    prof_end(g->ctx, PROF_ROWS, 0.0, 0.0);
}

void apply_operator_group(const std::vector<OpInput> &items) {
    // the folded tensor-core contractions that can share a launch: same context,
    // same product count, distinct geometries
    std::vector<size_t> grp;
    for (size_t i = 0; i < items.size(); ++i) {
        const OpInput &it = items[i];
        if (it.b.count == 0 || !(it.how == Contraction::TC3 || it.how == Contraction::TC1) ||
            !tc_folds_operator(it.g))
            continue;
        bool ok = true;
        for (size_t k : grp)
            ok = ok && items[k].g != it.g && items[k].g->ctx == it.g->ctx && items[k].how == it.how;
        if (ok) grp.push_back(i);
    }
    if (grp.size() < 2) {
        for (const OpInput &it : items) apply_operator(it.g, it.b, it.X, it.Y, it.work, it.how, it.presplit);
        return;
    }
    plx_ctx *ctx = items[grp[0]].g->ctx;
    std::vector<TcItem> ti;
    double flops = 0.0, bytes = 0.0;
    for (size_t k : grp) {
        const OpInput &it = items[k];
        ti.push_back(tc_item(it.g, it.b, it.X, it.Y, it.work, it.how, it.presplit));
        const double nn = (double)it.g->n_var;
        flops += 2.0 * nn * nn * 2.0 * it.b.count;
        bytes += tc_bytes(it.g, it.how, it.b.count);
    }
    prof_begin(ctx);
    tc_contract_group(ti);
    prof_end(ctx, PROF_TC, flops, bytes);
    for (size_t j = 0; j < grp.size(); ++j) {
        const OpInput &it = items[grp[j]];
        folded_finish(it.g, it.b, ti[j].S, it.Y);
    }
    for (size_t i = 0; i < items.size(); ++i)
        if (std::find(grp.begin(), grp.end(), i) == grp.end()) {
            const OpInput &it = items[i];
            apply_operator(it.g, it.b, it.X, it.Y, it.work, it.how, it.presplit);
        }
}

void rhs_batch(plx_geom *g, const OpBatch &b, const int32_t *d_pol, double *Bout) {
    if (b.count == 0) return;
    if (is_bem(g)) {
        bem_rhs(g, b, d_pol, Bout);
        return;
    }
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int N = g->n_atoms, nv = g->n_var;
    double mn[3] = {0, 0, 0};
    if (g->rhs_potential) {
        for (int k = 0; k < 3; ++k) {
            mn[k] = g->coord[k];
            for (int i = 0; i < N; ++i) mn[k] = std::min(mn[k], g->coord[k + 3 * i]);
        }
    }
    DevArray<double> V;
    V.alloc(ctx, (size_t)b.count * 2 * nv);
    potential_kernel<<<dim3(n_blocks(nv, 256), b.count), 256, 0, st>>>(
        N, nv, b.count, d_pol, g->d_pos.p, g->e0, g->rhs_potential, mn[0], mn[1], mn[2], V.p);
    ctx->launches++;
    // b_q = -Kop(w) V  (rhs_module.f90:140-390); no diagonal term
    DevArray<double> Vt;
    if (charges_by_column(g, b.count)) {
        try {
            Vt.alloc(ctx, (size_t)b.count * 2 * N);
        } catch (const Error &) {                     // no room: the row form needs none
        }
    }
    charge_part(g, b, V.p, V.p, Bout, -1.0, 0, Vt.p);
    if (g->model == PLX_WFQFMU) {
        dim3 gm(n_blocks(3LL * N, 256), b.count);
        rhs_dipole<<<gm, 256, 0, st>>>(N, nv, b.count, d_pol, g->e0, Bout);
        ctx->launches++;
    }
    PLX_CHECK_CUDA(cudaGetLastError());
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));
}

}  // namespace plx
