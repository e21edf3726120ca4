// Conductance folded into the interaction matrix, once per geometry:
//   A0[i][k] = sum_j c_ij (T[j][k] - T[i][k]),   i a charge row,
// with c_ij = K_ij for one atom type (the charge rows of (K - P) T, update_y_q of
// matrix_module.f90:1011-1098, applied to T itself) and 1/2 (K_ij + K_ji) for alloys (the
// w-independent part of 1/2 (K + (w_j/w_i) K^T)).
//
// A sparse (540 entries a row) times dense product.  A thread per element, walking its
// row's entries, read 2 x 10^11 elements of T through L1 for 10,473 atoms: 140 ms,
// 13% of a spectrum of that sphere.  Here the rows are taken in clusters of 32 atoms
// close in space (a Z-order curve): their neighbour lists overlap, so the cluster's
// coefficients are a dense (32 x union) block, about 1,400 columns of which a row uses
// 540, and a warp multiplies it with the union's rows of T on the FP64 matrix
// instruction, 8 rows x 4 neighbours at a time; tiles without an entry (the union
// follows the curve too, so four neighbours in a row lie together) are skipped.  Each
// element of T is read once per cluster.  The differences are taken against the
// cluster's first atom, t = T[j] - T[ref], and T[i] enters as
//   sum_j c_ij t_j - (sum_j c_ij) (T[i] - T[ref]),
// so that, as in the formula, only differences of neighbouring potentials are summed (in
// FP64, then split to the operand's 16 bits).  10,473 atoms, 41,892 columns: 140 -> 44 ms.
#include <algorithm>
#include <cmath>
#include <numeric>

#include "dmma.cuh"
#include "operand.cuh"
#include "pair_tiles.cuh"
#include "plx_internal.h"

namespace plx {

namespace {

constexpr int kCluster = 32;                         // rows of a cluster
constexpr size_t kFoldBytes = size_t(32) << 20;      // coefficients held at a time (at least one cluster's)

// Union of the neighbours of a cluster's rows as bits in curve order, in shared memory.
__device__ __forceinline__ void union_bits(int words, int c, const int32_t *__restrict__ rows,
                                           const int32_t *__restrict__ rank, const int32_t *__restrict__ rowptr,
                                           const int32_t *__restrict__ col, uint32_t *bits) {
    for (int w = threadIdx.x; w < words; w += blockDim.x) bits[w] = 0u;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = warp; r < kCluster; r += blockDim.x >> 5) {
        const int i = rows[c * kCluster + r];
        if (i < 0) continue;
        for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32) {
            const int k = rank[col[e]];
            atomicOr(&bits[k >> 5], 1u << (k & 31));
        }
    }
    __syncthreads();
}

// Number of union entries of every cluster.
__global__ void union_count(int words, const int32_t *__restrict__ rows, const int32_t *__restrict__ rank,
                            const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col,
                            int32_t *__restrict__ count) {
    extern __shared__ uint32_t bits[];
    __shared__ int total;
    if (threadIdx.x == 0) total = 0;
    union_bits(words, blockIdx.x, rows, rank, rowptr, col, bits);
    int s = 0;
    for (int w = threadIdx.x; w < words; w += blockDim.x) s += __popc(bits[w]);
    atomicAdd(&total, s);
    __syncthreads();
    if (threadIdx.x == 0) count[blockIdx.x] = total;
}

// The rows of T of the union's atoms (map: row of an atom, the atom itself when null;
// padded to fours with the cluster's first atom, coefficient zero) and the coefficients
// C[union entry][32 rows], zeroed before; row sums of the coefficients.
__global__ void union_fill(int words, int c0, int hetero, const int32_t *__restrict__ rows,
                           const int32_t *__restrict__ order, const int32_t *__restrict__ rank,
                           const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col,
                           const double *__restrict__ kval, const double *__restrict__ ktval,
                           const int32_t *__restrict__ map, const int32_t *__restrict__ off,
                           int32_t *__restrict__ list, double *__restrict__ C, double *__restrict__ csum) {
    extern __shared__ uint32_t bits[];
    int *prefix = reinterpret_cast<int *>(bits + words);         // set bits before a word
    const int c = c0 + blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    union_bits(words, c, rows, rank, rowptr, col, bits);
    if (warp == 0) {
        int base = 0;
        for (int w0 = 0; w0 < words; w0 += 32) {
            const int w = w0 + lane, v = w < words ? __popc(bits[w]) : 0;
            int s = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += t;
            }
            if (w < words) prefix[w] = base + s - v;
            base += __shfl_sync(0xffffffffu, s, 31);
        }
        // the padding
        const int o = off[blockIdx.x], end = off[blockIdx.x + 1] - off[0];
        const int first = map ? map[rows[c * kCluster]] : rows[c * kCluster];
        for (int u = o - off[0] + base + lane; u < end; u += 32) list[u] = first;
    }
    __syncthreads();
    const int o = off[blockIdx.x] - off[0];
    for (int w = threadIdx.x; w < words; w += blockDim.x) {
        uint32_t m = bits[w];
        int u = o + prefix[w];
        while (m) {
            const int b = __ffs(m) - 1;
            m &= m - 1;
            const int atom = order[32 * w + b];
            list[u++] = map ? map[atom] : atom;
        }
    }
    for (int r = warp; r < kCluster; r += blockDim.x >> 5) {
        const int i = rows[c * kCluster + r];
        double s = 0.0;
        if (i >= 0)
            for (int e = rowptr[i] + lane; e < rowptr[i + 1]; e += 32) {
                const int k = rank[col[e]];
                const double v = hetero ? 0.5 * (kval[e] + ktval[e]) : kval[e];
                const int u = o + prefix[k >> 5] + __popc(bits[k >> 5] & ((1u << (k & 31)) - 1));
                C[(int64_t)u * kCluster + r] = v;
                s += v;
            }
#pragma unroll
        for (int q = 16; q > 0; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
        if (lane == 0) csum[blockIdx.x * kCluster + r] = s;
    }
}

constexpr int kFoldNT = 4;                           // 8-column tiles of a warp
constexpr int kFoldCols = 4 * 8 * kFoldNT;           // columns of a block

__global__ void __launch_bounds__(128, 4) fold_clusters(int n, int c0, const int32_t *__restrict__ map,
                                                        const int32_t *__restrict__ rows,
                                                        const int32_t *__restrict__ off,
                                                        const int32_t *__restrict__ list,
                                                        const double *__restrict__ C, const double *__restrict__ csum,
                                                        const double *__restrict__ T, FoldTarget out) {
    constexpr int MT = kCluster / 8, NT = kFoldNT, D = 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kk = lane & 3, g = lane >> 2;
    const int col0 = blockIdx.y * kFoldCols + warp * 8 * NT;
    if (col0 >= n) return;
    const int *row = rows + (int64_t)(c0 + blockIdx.x) * kCluster;
    const int u0 = off[blockIdx.x] - off[0], u1 = off[blockIdx.x + 1] - off[0];
    auto t_row = [&](int i) { return T + (int64_t)(map ? map[i] : i) * n; };
    const double *Tref = t_row(row[0]);
    double t0[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) t0[t] = col0 + 8 * t + g < n ? __ldg(Tref + col0 + 8 * t + g) : 0.0;
    double acc[MT][NT][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
    double a[D][MT], b[D][NT];
    auto load = [&](int s, int u) {
        if (u >= u1) return;                         // the same for the warp (padded to fours)
        const double *Tj = T + (int64_t)__ldg(list + u + kk) * n + col0 + g;
#pragma unroll
        for (int t = 0; t < NT; ++t) b[s][t] = col0 + 8 * t + g < n ? __ldg(Tj + 8 * t) : 0.0;
        const double *Cu = C + (int64_t)(u + kk) * kCluster + g;
#pragma unroll
        for (int m = 0; m < MT; ++m) a[s][m] = __ldg(Cu + 8 * m);
    };
#pragma unroll
    for (int s = 0; s < D; ++s) load(s, u0 + 4 * s);
    for (int u = u0; u < u1; u += 4 * D) {
#pragma unroll
        for (int s = 0; s < D; ++s) {
            if (u + 4 * s < u1) {
                double d[NT];
#pragma unroll
                for (int t = 0; t < NT; ++t) d[t] = b[s][t] - t0[t];
#pragma unroll
                for (int m = 0; m < MT; ++m)
                    if (__any_sync(0xffffffffu, a[s][m] != 0.0)) {
#pragma unroll
                        for (int t = 0; t < NT; ++t) dmma(acc[m][t], a[s][m], d[t]);
                    }
            }
            load(s, u + 4 * D + 4 * s);
        }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        const int i = row[8 * m + g];
        if (i < 0) continue;
        const double cs = csum[blockIdx.x * kCluster + 8 * m + g];
        const double *Ti = t_row(i);
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int c = col0 + 8 * t + 2 * kk + v;
                if (c >= n) continue;
                const double x = fma(-cs, __ldg(Ti + c) - __ldg(Tref + c), acc[m][t][v]);
                split_store(x, a_tiled(i, c, out.ktiles), reinterpret_cast<__nv_bfloat16 *>(out.hi),
                            reinterpret_cast<__nv_bfloat16 *>(out.lo));
            }
    }
}

// Atoms along a Z-order curve over cells a nearest-neighbour distance wide.
std::vector<int32_t> curve_order(const plx_geom *g) {
    const int N = g->n_atoms;
    double h = 0.0, lo[3];
    for (double r : g->r0)
        if (r > 0.0 && std::isfinite(r)) h = h == 0.0 ? r : std::min(h, r);
    for (int k = 0; k < 3; ++k) {
        lo[k] = g->coord[k];
        double hi = lo[k];
        for (int i = 1; i < N; ++i) {
            lo[k] = std::min(lo[k], g->coord[k + 3 * (size_t)i]);
            hi = std::max(hi, g->coord[k + 3 * (size_t)i]);
        }
        h = std::max(h, (hi - lo[k]) / double(1 << 20));         // 21 bits a coordinate
    }
    std::vector<uint64_t> key(N, 0);
    if (h > 0.0 && std::isfinite(h))
        for (int i = 0; i < N; ++i)
            for (int k = 0; k < 3; ++k) {
                const double q = std::floor((g->coord[k + 3 * (size_t)i] - lo[k]) / h);
                uint64_t v = q >= 0.0 && q < double(1 << 21) ? (uint64_t)q : 0;
                for (int b = 0; v; ++b, v >>= 1) key[i] |= (v & 1) << (3 * b + k);
            }
    std::vector<int32_t> order(N);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return key[a] < key[b]; });
    return order;
}

// Charge rows of T of the listed atoms: a thread per pair writes the charge and the three
// dipole elements.
__global__ void charge_rows_gen(int N, int n, int nt, int fmu, const int32_t *__restrict__ atoms,
                                const double *__restrict__ pos, const double *__restrict__ par,
                                const int32_t *__restrict__ type, const PairWidths *__restrict__ widths,
                                double *__restrict__ Tw) {
    const int j = blockIdx.y * blockDim.x + threadIdx.x;
    if (j >= N) return;
    const int i = atoms[blockIdx.x];
    double *o = Tw + (int64_t)blockIdx.x * n;
    double q = 0.0, m[3] = {0.0, 0.0, 0.0};
    if (i == j) {
        q = par[2 * N + i];
    } else {
        const double dx = pos[i] - pos[j], dy = pos[N + i] - pos[N + j], dz = pos[2 * N + i] - pos[2 * N + j];
        const int ti = type[i], tj = type[j];
        if (!fmu) {
            q = plx_pair_qq_w(dx, dy, dz, widths[ti + nt * tj]);
        } else {
            PairTile t;
            plx_pair_tile_w(dx, dy, dz, widths[ti + nt * tj], ti == tj, t);
            q = t.qq;
            for (int k = 0; k < 3; ++k) m[k] = t.qm[k];
        }
    }
    o[j] = q;
    if (fmu)
        for (int k = 0; k < 3; ++k) o[N + 3 * j + k] = m[k];
}

// Folds the clusters of d_rows (nc of them) from rows of T.
void fold_batch(plx_geom *g, int nc, const int32_t *d_rows, const int32_t *d_order, const int32_t *d_rank,
                const int32_t *d_map, const double *T, const FoldTarget &out) {
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int N = g->n_atoms, n = g->n_var, words = (N + 31) / 32;
    const size_t smem = (size_t)words * 8;
    DevArray<int32_t> d_count;
    d_count.alloc(ctx, nc);
    union_count<<<nc, 256, smem, st>>>(words, d_rows, d_rank, g->d_rowptr.p, g->d_col.p, d_count.p);
    ctx->launches++;
    PLX_CHECK_CUDA(cudaGetLastError());
    std::vector<int32_t> count(nc), off(nc + 1, 0);
    PLX_CHECK_CUDA(cudaMemcpyAsync(count.data(), d_count.p, (size_t)nc * 4, cudaMemcpyDeviceToHost, st));
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));
    for (int c = 0; c < nc; ++c) off[c + 1] = off[c] + (count[c] + 3) / 4 * 4;
    DevArray<int32_t> d_off, d_list;
    DevArray<double> d_C, d_csum;
    d_off.alloc(ctx, nc + 1);
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_off.p, off.data(), (size_t)(nc + 1) * 4, cudaMemcpyHostToDevice, st));
    int most = (int)(kFoldBytes / (kCluster * sizeof(double)));
    for (int c0 = 0; c0 < nc;) {
        int c1 = c0 + 1;
        while (c1 < nc && off[c1 + 1] - off[c0] <= most) ++c1;
        const size_t len = std::max(1, off[c1] - off[c0]);
        if (d_list.n < len || d_C.n < len * kCluster) {
            try {
                d_list.alloc(ctx, len);
                d_C.alloc(ctx, len * kCluster);
            } catch (const Error &) {                 // little room: smaller batches, down to a cluster
                d_list.release();
                d_C.release();
                if (c1 == c0 + 1) throw;
                most /= 4;
                continue;
            }
        }
        if (d_csum.n < (size_t)(c1 - c0) * kCluster) d_csum.alloc(ctx, (size_t)(c1 - c0) * kCluster);
        PLX_CHECK_CUDA(cudaMemsetAsync(d_C.p, 0, len * kCluster * 8, st));
        union_fill<<<c1 - c0, 256, smem, st>>>(words, c0, g->n_types > 1, d_rows, d_order, d_rank, g->d_rowptr.p,
                                               g->d_col.p, g->d_kval.p, g->d_ktval.p, d_map, d_off.p + c0, d_list.p,
                                               d_C.p, d_csum.p);
        // clusters vary fastest over the grid: the blocks running together share their rows of T in L2
        fold_clusters<<<dim3(c1 - c0, n_blocks(n, kFoldCols)), 128, 0, st>>>(n, c0, d_map, d_rows, d_off.p + c0, d_list.p,
                                                                            d_C.p, d_csum.p, T, out);
        ctx->launches += 2;
        PLX_CHECK_CUDA(cudaGetLastError());
        c0 = c1;
    }
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));     // host vectors feed the copies above
}

}  // namespace

void fold_charge_rows(plx_geom *g, const FoldTarget &out) {
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int N = g->n_atoms, n = g->n_var;
    if ((size_t)((N + 31) / 32) * 8 > 200 * 1024) throw Error(PLX_ERR_UNSUPPORTED, "too many atoms for the folded operand");
    const std::vector<int32_t> order = curve_order(g);
    const int nc = n_blocks(N, kCluster);
    std::vector<int32_t> rank(N), rows(order);
    for (int k = 0; k < N; ++k) rank[order[k]] = k;
    rows.resize((size_t)nc * kCluster, -1);
    DevArray<int32_t> d_order, d_rank, d_rows;
    d_order.alloc(ctx, N);
    d_rank.alloc(ctx, N);
    d_rows.alloc(ctx, rows.size());
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_order.p, order.data(), (size_t)N * 4, cudaMemcpyHostToDevice, st));
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_rank.p, rank.data(), (size_t)N * 4, cudaMemcpyHostToDevice, st));
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_rows.p, rows.data(), rows.size() * 4, cudaMemcpyHostToDevice, st));
    once_per_device(reinterpret_cast<const void *>(union_fill), ctx->device, [] {
        PLX_CHECK_CUDA(cudaFuncSetAttribute(union_count, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        PLX_CHECK_CUDA(cudaFuncSetAttribute(union_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
    });
    if (g->has_T) {
        fold_batch(g, nc, d_rows.p, d_order.p, d_rank.p, nullptr, g->d_T.p, out);
        return;
    }
    // matrix-free: batches of clusters whose atoms and neighbours are at most max_rows (about
    // 6 GB of generated rows; a cluster that needs more gets them)
    std::vector<int32_t> rowptr(N + 1), col((size_t)g->nnz);
    PLX_CHECK_CUDA(cudaMemcpyAsync(rowptr.data(), g->d_rowptr.p, (N + 1) * 4, cudaMemcpyDeviceToHost, st));
    if (g->nnz) PLX_CHECK_CUDA(cudaMemcpyAsync(col.data(), g->d_col.p, g->nnz * 4, cudaMemcpyDeviceToHost, st));
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));
    const size_t max_rows = std::max<size_t>(64, (size_t)(6.0e9 / (8.0 * (double)n)));
    DevArray<double> Tw;
    DevArray<int32_t> d_atoms, d_map;
    d_map.alloc(ctx, N);
    std::vector<int32_t> map(N, -1), atoms, more;
    for (int c0 = 0; c0 < nc;) {
        atoms.clear();
        std::fill(map.begin(), map.end(), -1);
        int c1 = c0;
        for (; c1 < nc; ++c1) {
            more.clear();
            auto take = [&](int a) {
                if (map[a] < 0) {
                    map[a] = (int32_t)(atoms.size() + more.size());
                    more.push_back(a);
                }
            };
            for (int r = 0; r < kCluster; ++r) {
                const int i = rows[(size_t)c1 * kCluster + r];
                if (i < 0) continue;
                take(i);
                for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) take(col[e]);
            }
            if (c1 > c0 && atoms.size() + more.size() > max_rows) {
                for (int a : more) map[a] = -1;
                break;
            }
            atoms.insert(atoms.end(), more.begin(), more.end());
        }
        if (Tw.n < atoms.size() * n) {
            Tw.alloc(ctx, atoms.size() * n);
            d_atoms.alloc(ctx, atoms.size());
        }
        PLX_CHECK_CUDA(cudaMemcpyAsync(d_atoms.p, atoms.data(), atoms.size() * 4, cudaMemcpyHostToDevice, st));
        PLX_CHECK_CUDA(cudaMemcpyAsync(d_map.p, map.data(), (size_t)N * 4, cudaMemcpyHostToDevice, st));
        charge_rows_gen<<<dim3((unsigned)atoms.size(), n_blocks(N, 128)), 128, 0, st>>>(
            N, n, g->n_types, g->model == PLX_WFQFMU, d_atoms.p, g->d_pos.p, g->d_par.p, g->d_type.p, g->d_widths.p, Tw.p);
        ctx->launches++;
        fold_batch(g, c1 - c0, d_rows.p + (size_t)c0 * kCluster, d_order.p, d_rank.p, d_map.p, Tw.p, out);
        c0 = c1;
    }
}

}  // namespace plx
