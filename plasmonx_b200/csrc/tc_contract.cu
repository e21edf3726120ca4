// Tensor-core T contraction for the mixed-precision solve (sm_100a, tcgen05).
//
// S = T X for a batch of R real columns, with T (n x n, symmetric) and X split
// into BF16 high and low parts, T = Th + Tl, X = Xh + Xl, and
//     S = Th Xh + Th Xl + Tl Xh        (FP32 accumulation in tensor memory),
// i.e. every product carries ~16 significant bits of each operand; the dropped
// Tl Xl term is below 2^-16 of the result.  The result is written as FP64 so the
// rest of the operator (conductance rows, frequency diagonal) stays unchanged.
//
// GEMM mapping (all operands K-major, the layout tcgen05 reads natively):
//   A = T   rows m of T, contiguous along k         (M = n_var)
//   B = X^T column c of X, contiguous along k        (N = R real columns)
//   D = TMEM accumulators 128 x BN (FP32), lane = row m, column = c
// One CTA computes a 256 x BN tile of S as two 128-row accumulators (TMEM
// columns [0, BN) and [BN, 2 BN)) that share every B tile, which halves the
// B traffic from L2 per row of T.  Six warps: warps 0-3 drain TMEM in the
// epilogue, one thread of warp 4 issues the loads and one of warp 5 the MMAs.
// Operand tiles are 32 elements (64 bytes) deep along k and are
// loaded by TMA with the 64-byte swizzle that the UMMA descriptors describe;
// the small stages allow 3-6 of them in flight with three products, 7 or 8 with one.
// Every wait on an mbarrier is bounded.  The pipeline waits use the context's
// limit (plx_set_wait_limit); a CTA whose wait runs out records an error code
// and gives up, in this order: the MMA issuer still commits `drained`, which
// arrives only when every MMA it has issued has finished; all threads wait for
// it, so no MMA reads shared memory or writes tensor memory after that point;
// the producer then waits for the loads it has issued to land, so no copy
// writes into shared memory after the CTA exits; then the tensor memory is
// freed and the CTA returns without storing a result.  These clean-up waits
// use their own, long limit (kDrainLimit), never the pipeline limit.  If one of
// them runs out as well (a copy or an MMA that never completes: the hardware
// has stopped answering) the CTA records that error too and exits anyway; the
// call then fails and nothing it wrote is used.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>

#include "operand.cuh"
#include "pair_tiles.cuh"
#include "pdl.cuh"
#include "plx_internal.h"

namespace plx {

namespace {

constexpr int kUM = kBM / 2;      // rows per tcgen05.mma (TMEM lanes): two accumulators share every B tile
constexpr int kLdAlign = 64;      // k padding of the split operands (zeros)
constexpr int kUmmaK = 16;        // k per tcgen05.mma (kind::f16)
constexpr uint32_t kDrainLimit = 1u << 22;  // clean-up waits after an abort (seconds at most)
constexpr int kSmemBudget = 227 * 1024 - 1024 - 256;   // pipeline stages (after alignment and barriers)

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: returns false when `limit` polls pass, or early when another
// thread of the CTA has raised `abort`; records `code` in *err on failure.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint32_t limit, volatile int *abort,
                                          int *err, int code) {
    for (uint32_t it = 0; it < limit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if (abort && (it & 255u) == 255u && *abort) return false;
    }
    if (err) atomicCAS(err, 0, code);
    return false;
}

// Plain bulk copy of `bytes` contiguous bytes into shared memory (addresses
// 16-byte aligned, size a multiple of 16), completing on `bar`.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tma_load_2d(const CUtensorMap *map, uint64_t *bar, void *dst, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// UMMA shared-memory descriptor, K-major operand with the 64-byte swizzle:
// 8-row x 64-byte swizzle atoms stacked every 512 bytes (stride byte offset),
// leading byte offset 16 bytes (unused for this layout), descriptor version 1,
// layout type 4 (64-byte swizzle) in bits [61,64).
__device__ __forceinline__ uint64_t umma_desc_sw64(const void *smem) {
    uint64_t addr = smem_u32(smem);
    uint64_t d = 0;
    d |= (addr >> 4) & 0x3FFFull;           // start address, bits [0,14)
    d |= (uint64_t)(16 >> 4) << 16;         // leading byte offset, bits [16,30)
    d |= (uint64_t)(512 >> 4) << 32;        // stride byte offset, bits [32,46)
    d |= (uint64_t)1 << 46;                 // version, bits [46,48)
    d |= (uint64_t)4 << 61;                 // layout: 64-byte swizzle
    return d;
}

// Instruction descriptor, kind::f16: BF16 x BF16 -> FP32, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4)                        // D format F32
           | (1u << 7)                      // A format BF16
           | (1u << 10)                     // B format BF16
           | ((uint32_t)(N >> 3) << 17)     // N / 8
           | ((uint32_t)(M >> 4) << 24);    // M / 16
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

// Work of one launch: the output tiles (256 rows x bn columns, column tile
// fastest so that the tiles sharing one row block of an operand run side by
// side and its second read comes from L2) of one or several groups -- a group
// is one contraction S = A X of one geometry -- in one list, the groups ordered
// by decreasing k length.  The first `full` tiles (whole waves of the chip) are
// computed whole, one CTA each.  The k-tiles of the remaining tiles, end to end,
// are dealt to the CTAs of the last wave in equal runs of `run` k-tiles (at least
// kMinRun): a run covers the end of one tile, perhaps whole small tiles, and the
// beginning of another.  A tile that lies in one run is stored like a whole one;
// the others leave FP32 partial sums ([column][row], slot = tile + CTA index, which
// no two of them share), added in k order by reduce_pieces.
//
// The operand is streamed once whatever the split, so the launch is bound by HBM
// (by L2 for operands that fit it) as long as every SM has the same share.  Splitting
// each remaining tile into sms / remaining equal pieces left 38 SMs of 148 idle at 55
// tiles (13,528 unknowns: 156 us a launch, now 121 us) and 24 at 31 tiles (7,844
// unknowns: 51.7 -> 47 us); grouped launches ran whole tiles only, 30 CTAs for six
// geometries of 143 to 2,700 unknowns (25.9 -> 9.2 us).
constexpr int kMaxGroups = 6;
// k-tiles a CTA at least.  Six small geometries: 11.2 us a launch with 8, 9.2 with 4, 8.4
// with 2, which costs the pieces another microsecond.
constexpr int kMinRun = 4;
constexpr int kThreadsTc = 192;

// The rest of an operator row after the contraction, applied where its sums are
// complete: Y = S + D(w) X for the first n rows (D(w): -z(w) of the atom's type on
// charge rows, sum_t f_t,i / alpha_t(w) on dipole rows; the BEM's z(w) with N = n,
// nt = 1, type = null).  Rows beyond n go to S as without it.
struct TcRows {
    int n, N, nt;
    const int32_t *freq, *type;
    const Cplx *dq;
    const double *frac;
    const Cplx *inv_alpha;
    const double *X;
    double *Y;                  // null: no rows, S alone
};
struct TcGroup {
    int M, R, bn, ktiles;       // rows, real columns, column tile, k-tiles (32 deep)
    int ctiles;                 // column tiles
    int tile0;                  // index of the group's first tile in the launch's list
    int unit0;                  // k-tiles of the split tiles before the group
    const uint8_t *ah, *al;     // A high / low, tile-ordered and pre-swizzled (16 KB per stage tile)
    double *S;                  // [R][M] FP64
    TcRows rows;
};
struct TcLaunch {
    CUtensorMap map[kMaxGroups][2];   // X high, X low (A goes by bulk copy)
    TcGroup grp[kMaxGroups];
    int ngroups, tiles;
    int full;                   // tiles computed whole, one CTA each
    int run, units;             // k-tiles a CTA of the split tiles takes, and their number
    float *P;                   // partial sums, slots of 256 x bn_max
    int stages;                 // pipeline depth
    int bn_max;                 // shared-memory / tensor-memory sizing
    uint32_t wait_limit;
    int *err;                   // first bounded wait that ran out: the first group's geometry's word, the launch's only one
};

// A piece of work of a CTA: k-tiles [kt0, kt0 + nk) of a group's tile.
struct TcSeg {
    int gi, tile, kt0, nk, slot;     // slot < 0: the whole tile
};

// Group of tile t of the launch's list.
__device__ __forceinline__ int group_of_tile(const TcLaunch &p, int t) {
    int g = 0;
    while (g + 1 < p.ngroups && t >= p.grp[g + 1].tile0) ++g;
    return g;
}

// First split tile of a group (index within the group).
__device__ __forceinline__ int first_split(const TcLaunch &p, int g) { return max(0, p.full - p.grp[g].tile0); }

// The segments of a CTA in order: call with u = start of its range, advances u.
__device__ __forceinline__ TcSeg next_segment(const TcLaunch &p, int cta, int &u, int uend) {
    TcSeg s;
    if (cta < p.full) {
        s.gi = group_of_tile(p, cta);
        s.tile = cta - p.grp[s.gi].tile0;
        s.kt0 = 0;
        s.nk = p.grp[s.gi].ktiles;
        s.slot = -1;
        u = uend;
        return s;
    }
    int g = 0;
    while (g + 1 < p.ngroups && u >= p.grp[g + 1].unit0) ++g;
    const int kt = p.grp[g].ktiles, rem = u - p.grp[g].unit0, local = rem / kt;
    s.gi = g;
    s.tile = first_split(p, g) + local;
    s.kt0 = rem - local * kt;
    s.nk = min(kt - s.kt0, uend - u);
    s.slot = s.nk == kt ? -1 : p.grp[g].tile0 + s.tile - p.full + (cta - p.full);
    u += s.nk;
    return s;
}

// Stores the complete sums s of real columns c .. c + 2 NP - 1 (NP complex columns,
// those inside the batch) at row r.  All its loads go out before the first store: one
// column after the other, each behind the previous one's store, took 50 us of a
// 713 us launch at 48 columns.
template <int NP>
__device__ __forceinline__ void store_columns(const TcGroup &G, int r, int c, const double (&s)[2 * NP]) {
    const TcRows &q = G.rows;
    if (!(q.Y && r < q.n)) {
#pragma unroll
        for (int k = 0; k < 2 * NP; ++k)
            if (c + k < G.R) G.S[(int64_t)(c + k) * G.M + r] = s[k];
        return;
    }
    Cplx d[NP];
    double x[2 * NP];
    int f[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        const bool in = c + 2 * k < G.R;
        f[k] = in ? __ldg(q.freq + (c >> 1) + k) : 0;
        const int64_t o = (int64_t)(c + 2 * k) * q.n + r;
        x[2 * k] = in ? __ldg(q.X + o) : 0.0;
        x[2 * k + 1] = in ? __ldg(q.X + o + q.n) : 0.0;
        d[k] = {0.0, 0.0};
    }
    if (r < q.N) {
        const double2 *dq = reinterpret_cast<const double2 *>(q.dq) + (q.type ? __ldg(q.type + r) : 0);
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            const double2 v = __ldg(dq + q.nt * f[k]);
            d[k] = {v.x, v.y};
        }
    } else {
        const double *frac = q.frac + (int64_t)q.nt * ((r - q.N) / 3);
        for (int t = 0; t < q.nt; ++t) {
            const double fr = __ldg(frac + t);
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const double2 v = __ldg(reinterpret_cast<const double2 *>(q.inv_alpha) + t + q.nt * f[k]);
                d[k].re += fr * v.x;
                d[k].im += fr * v.y;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NP; ++k)
        if (c + 2 * k < G.R) {
            const int64_t o = (int64_t)(c + 2 * k) * q.n + r;
            q.Y[o] = s[2 * k] + d[k].re * x[2 * k] - d[k].im * x[2 * k + 1];
            q.Y[o + q.n] = s[2 * k + 1] + d[k].re * x[2 * k + 1] + d[k].im * x[2 * k];
        }
}

// Bytes of one pipeline stage: the A and X tiles its products read -- high and
// low parts for three products, the high parts alone for one (whose stages are
// then half as large and twice as many fit).
__host__ __device__ constexpr int tc_stage_bytes(int bn, int nprod) {
    return (nprod > 1 ? 2 : 1) * (kBM * kBK * 2 + bn * kBK * 2);
}

template <int NPROD>
__global__ void __launch_bounds__(kThreadsTc, 1) tc_contract_kernel(const __grid_constant__ TcLaunch p) {
    const int cta = (int)blockIdx.x;
    const int u0 = cta < p.full ? 0 : (cta - p.full) * p.run;
    const int uend = cta < p.full ? 1 : min(p.units, u0 + p.run);
    const int STAGES = p.stages;
    const int kStage = tc_stage_bytes(p.bn_max, NPROD);
    const int kA = kBM * kBK * 2;
    const uint32_t wait_limit = p.wait_limit;
    // an accumulator set is two accumulators (rows m0.. and m0 + 128..) of bn_max columns
    // (a multiple of 32); two sets where they fit the 512 TMEM columns, so that a
    // segment's products start while the previous one is stored
    const int set_cols = 2 * p.bn_max;
    const int nbuf = 2 * set_cols <= 512 ? 2 : 1;
    const int need_cols = nbuf * set_cols;
    const uint32_t tmem_cols = need_cols <= 64 ? 64 : (need_cols <= 128 ? 128 : (need_cols <= 256 ? 256 : 512));
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(base + STAGES * kStage);
    uint64_t *empty = full + STAGES;
    uint64_t *done = empty + STAGES;          // [2]: a set's sums are complete
    uint64_t *freed = done + 2;               // [2]: a set has been read out
    uint64_t *drained = freed + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drained + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    int *err = p.err;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&done[s], 1);
            mbar_init(&freed[s], 128);
        }
        mbar_init(drained, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_sync();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    // a stage holds A high (A low), X high (X low); the low parts only for NPROD > 1.  The
    // issuing threads keep stage, phase and addresses as running values: their loop is the
    // launch's limit at few columns, and recomputing them (a division by the number of
    // stages among it) cost 640 cycles a k-tile against 32-64 per product (41,892
    // unknowns, 42 columns: one product 675 -> 509 us, three 1,077 -> 990 us, 6.9-7.1 TB/s)
    constexpr int kParts = NPROD > 1 ? 2 : 1;
    const int kX = kParts * kA, kXl = p.bn_max * kBK * 2;

    int issued = 0;     // loads issued by the producer
    if (threadIdx.x == 128) {
        // ---------------- TMA producer ----------------
        int u = u0, s = 0;
        uint32_t ph = 1;                      // a stage's first use finds its barrier free
        uint8_t *st = base;
        bool ok = true;
        while (u < uend && ok) {
            const TcSeg sg = next_segment(p, cta, u, uend);
            const TcGroup &G = p.grp[sg.gi];
            const CUtensorMap *mp = p.map[sg.gi];
            const int bn = G.bn, mtile = sg.tile / G.ctiles, n0 = (sg.tile % G.ctiles) * bn;
            // one product (NPROD = 1) reads only the high parts: half the operand bytes
            const uint32_t tx = (uint32_t)(NPROD > 1 ? 2 * kA + 2 * bn * kBK * 2 : kA + bn * kBK * 2);
            const size_t a0 = (size_t)(mtile * (int64_t)G.ktiles + sg.kt0) * kA;   // tile-ordered A
            const uint8_t *ah = G.ah + a0, *al = G.al + a0;
            int kx = sg.kt0 * kBK;
            for (int kt = 0; kt < sg.nk; ++kt) {
                if (!mbar_wait(&empty[s], ph, wait_limit, abort_flag, err, 1)) {
                    *abort_flag = 1;
                    ok = false;
                    break;
                }
                uint64_t *bar = &full[s];
                mbar_expect_tx(bar, tx);
                bulk_load(st, ah, kA, bar);
                if (NPROD > 1) bulk_load(st + kA, al, kA, bar);
                tma_load_2d(&mp[0], bar, st + kX, kx, n0);
                if (NPROD > 1) tma_load_2d(&mp[1], bar, st + kX + kXl, kx, n0);
                ah += kA;
                al += kA;
                kx += kBK;
                ++issued;
                st += kStage;
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                    st = base;
                }
            }
        }
    } else if (threadIdx.x == 160) {
        // ---------------- MMA issuer ----------------
        constexpr uint64_t kHalf = (uint64_t)(kUM * kBK * 2) >> 4;   // second 128 rows of an A tile
        // stage 0's descriptors; a stage, a part and a k step add to the address field
        const uint64_t d0 = umma_desc_sw64(base);
        const uint64_t dStage = (uint64_t)kStage >> 4, dLow = (uint64_t)kA >> 4, dX = (uint64_t)kX >> 4,
                       dXl = (uint64_t)kXl >> 4;
        int u = u0, s = 0;
        uint32_t ph = 0;
        uint64_t da = d0;
        bool ok = true;
        for (int seg = 0; u < uend && ok; ++seg) {
            const TcSeg sg = next_segment(p, cta, u, uend);
            const int buf = seg % nbuf;
            const uint32_t idesc = umma_idesc_bf16(kUM, p.grp[sg.gi].bn);
            if (seg >= nbuf && !mbar_wait(&freed[buf], ((seg / nbuf) - 1) & 1, wait_limit, abort_flag, err, 6)) {
                *abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t t0 = tmem + (uint32_t)(buf * set_cols), t1 = t0 + (uint32_t)p.bn_max;
            for (int kt = 0; kt < sg.nk; ++kt) {
                if (!mbar_wait(&full[s], ph, wait_limit, abort_flag, err, 2)) {
                    *abort_flag = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int kk = 0; kk < kBK / kUmmaK; ++kk) {
                    // advance 16 elements = 32 bytes = 2 descriptor units along k
                    const uint64_t a = da + ((uint64_t)(kk * kUmmaK * 2) >> 4), x = a + dX;
                    const uint32_t acc0 = (kt > 0 || kk > 0) ? 1u : 0u;
                    umma_bf16(t0, a, x, idesc, acc0);
                    umma_bf16(t1, a + kHalf, x, idesc, acc0);
                    if (NPROD > 1) {
                        umma_bf16(t0, a, x + dXl, idesc, 1u);
                        umma_bf16(t1, a + kHalf, x + dXl, idesc, 1u);
                        umma_bf16(t0, a + dLow, x, idesc, 1u);
                        umma_bf16(t1, a + dLow + kHalf, x, idesc, 1u);
                    }
                }
                umma_commit(&empty[s]);
                da += dStage;
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                    da = d0;
                }
            }
            if (ok) umma_commit(&done[buf]);
        }
        // always: arrives once every MMA issued above has completed (also after
        // an abort, so that nothing below frees memory an MMA still uses)
        umma_commit(drained);
    } else if (warp < 4) {
        // ---------------- epilogue: TMEM -> result, or the piece's partial (FP32) ----------------
        int u = u0;
        for (int seg = 0; u < uend; ++seg) {
            const TcSeg sg = next_segment(p, cta, u, uend);
            const TcGroup &G = p.grp[sg.gi];
            const int bn = G.bn, buf = seg % nbuf;
            const int m0 = sg.tile / G.ctiles * kBM, n0 = (sg.tile % G.ctiles) * bn;
            // one lane polls; the warp stays together, the loads below are warp-wide
            bool ok = true;
            if (lane == 0) ok = mbar_wait(&done[buf], (seg / nbuf) & 1, wait_limit, abort_flag, err, 3) && !*abort_flag;
            if (!__all_sync(0xffffffffu, ok)) {
                *abort_flag = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int h = 0; h < 2; ++h) {
                const int row = m0 + h * kUM + warp * 32 + lane;
#pragma unroll 1
                for (int c0 = 0; c0 < bn; c0 += 16) {
                    uint32_t v[16];
                    const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(buf * set_cols + h * p.bn_max + c0);
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                          "=r"(v[14]), "=r"(v[15])
                        : "r"(taddr));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (sg.slot >= 0) {
                        // partial of a split tile: [column][256 rows] FP32, every element written
                        float *pp = p.P + (int64_t)sg.slot * kBM * p.bn_max + (h * kUM + warp * 32 + lane);
#pragma unroll
                        for (int j = 0; j < 16; ++j) pp[(int64_t)(c0 + j) * kBM] = __uint_as_float(v[j]);
                    } else if (row < G.M) {
                        double s[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) s[j] = (double)__uint_as_float(v[j]);
                        store_columns<8>(G, row, n0 + c0, s);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&freed[buf]);
        }
    }
    __syncwarp();
    __syncthreads();
    // every MMA issued has finished before shared and tensor memory go
    if (!mbar_wait(drained, 0, kDrainLimit, nullptr, err, 4)) *abort_flag = 1;
    if (threadIdx.x == 128 && *abort_flag) {
        // let the loads already issued land before the CTA can exit: the last
        // phase of each stage (earlier phases completed before it was re-armed)
        for (int kt = issued > STAGES ? issued - STAGES : 0; kt < issued; ++kt)
            mbar_wait(&full[kt % STAGES], (kt / STAGES) & 1, kDrainLimit, nullptr, err, 5);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
    }
}

// Split tiles: the sum of a tile's FP32 pieces in k order (FP64 sums), stored like a
// whole tile.  One block per (split tile, eight columns), a thread per row: all its
// loads are independent (32 columns a block and thread: 14 us at 7,844 unknowns and
// 124 pieces, now 6.6 us with the diagonal rows that took 4.1 us in a launch of
// their own).
constexpr int kRedCols = 8;
__global__ void __launch_bounds__(kBM) reduce_pieces(const __grid_constant__ TcLaunch p) {
    pdl_sync();
    const int t = p.full + blockIdx.x;                       // index in the launch's list
    const int g = group_of_tile(p, t);
    const TcGroup &G = p.grp[g];
    const int tile = t - G.tile0;
    const int k0 = G.unit0 + (tile - first_split(p, g)) * G.ktiles;      // its k-tiles [k0, k0 + ktiles)
    const int f0 = k0 / p.run, f1 = (k0 + G.ktiles - 1) / p.run;         // CTAs that hold them
    if (f0 == f1) return;                                    // stored by its one CTA
    const int m0 = tile / G.ctiles * kBM, n0 = (tile % G.ctiles) * G.bn;
    const int r = threadIdx.x, c0 = blockIdx.y * kRedCols;
    if (m0 + r >= G.M || c0 >= G.bn) return;
    double a[kRedCols];
#pragma unroll
    for (int j = 0; j < kRedCols; ++j) a[j] = 0.0;
    for (int c = f0; c <= f1; ++c) {
        const float *pp = p.P + ((int64_t)(blockIdx.x + c) * p.bn_max + c0) * kBM + r;
#pragma unroll
        for (int j = 0; j < kRedCols; ++j) a[j] += (double)pp[(int64_t)j * kBM];
    }
    store_columns<kRedCols / 2>(G, m0 + r, n0 + c0, a);
}

// Row-major n x n FP64 matrix -> tiled BF16 pair; the output is walked in its
// own (contiguous) order.
__global__ void split_tiled(int n, int64_t ktiles, int64_t total, const double *__restrict__ in,
                            __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t kk = e % kBK, rr = (e / kBK) % kBM, tk = e / ((int64_t)kBK * kBM);
        const int64_t r = (tk / ktiles) * kBM + rr, k = (tk % ktiles) * kBK + kk;
        const double a = (r < n && k < n) ? in[r * n + k] : 0.0;
        split_store(a, tk * (int64_t)(kBM * kBK) + a_tile_pos(rr, kk), hi, lo);
    }
}

// Transposed (BEM: d_T[j][i] = D(i, j)): out(r, k) = in[k][r], through a
// shared-memory tile of 32 k x 256 r; grid (ktiles, mtiles).
__global__ void split_tiled_t(int n, int64_t ktiles, const double *__restrict__ in, __nv_bfloat16 *__restrict__ hi,
                              __nv_bfloat16 *__restrict__ lo) {
    __shared__ float tile[kBK][kBM + 1];
    const int64_t k0 = (int64_t)blockIdx.x * kBK, r0 = (int64_t)blockIdx.y * kBM;
    for (int e = threadIdx.x; e < kBK * kBM; e += blockDim.x) {
        const int kk = e / kBM, rr = e % kBM;                      // coalesced along r
        const int64_t k = k0 + kk, r = r0 + rr;
        tile[kk][rr] = (k < n && r < n) ? (float)in[k * n + r] : 0.0f;
    }
    __syncthreads();
    const int64_t base = ((int64_t)blockIdx.y * ktiles + blockIdx.x) * kBM * kBK;
    for (int e = threadIdx.x; e < kBK * kBM; e += blockDim.x) {   // contiguous output block
        const int rr = e / kBK, kk = e % kBK;
        float x = tile[kk][rr];
        __nv_bfloat16 h = __float2bfloat16_rn(x);
        hi[base + a_tile_pos(rr, kk)] = h;
        lo[base + a_tile_pos(rr, kk)] = __float2bfloat16_rn(x - __bfloat162float(h));
    }
}

// No stored T (on-the-fly geometries): the split generated from the pair
// formulas, one block per TMA box (256 rows x 32 k, contiguous output).
__global__ void split_tiled_gen(int N, int n, int fmu, int64_t ktiles, const double *__restrict__ pos,
                                const double *__restrict__ par, __nv_bfloat16 *__restrict__ hi,
                                __nv_bfloat16 *__restrict__ lo) {
    const int64_t k0 = (int64_t)blockIdx.x * kBK, r0 = (int64_t)blockIdx.y * kBM;
    const int64_t base = ((int64_t)blockIdx.y * ktiles + blockIdx.x) * kBM * kBK;
    for (int e = threadIdx.x; e < kBK * kBM; e += blockDim.x) {
        const int64_t r = r0 + e / kBK, k = k0 + e % kBK;
        const double a = (r < n && k < n) ? plx_t_element(N, fmu != 0, pos, par, r, k) : 0.0;
        split_store(a, base + a_tile_pos(e / kBK, e % kBK), hi, lo);
    }
}

// Rows of the folded operand that are rows of T, split like T: the dipole rows r < n
// and, after them, the charge rows of the interface atoms.  (The charge rows are folded
// in fold.cu.)
__global__ void copy_rows_split(int N, int n, int64_t ktiles, const double *__restrict__ T,
                                const int32_t *__restrict__ iface_atom, __nv_bfloat16 *__restrict__ hi,
                                __nv_bfloat16 *__restrict__ lo) {
    const int64_t r = N + (int64_t)blockIdx.x;
    const int64_t k = (int64_t)blockIdx.y * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int64_t src = r < n ? r : iface_atom[r - n];
    split_store(T[src * n + k], a_tiled(r, k, ktiles), hi, lo);
}

// The same rows without a stored T, a thread per pair of atoms: the dipole rows of atom i
// (or, beyond N, the charge row of interface atom i - N) against atom j, whose error
// functions and exponential are evaluated once for the pair's 12 (4) elements.
__global__ void pair_rows_split(int N, int n, int nt, int fmu, int64_t ktiles, const double *__restrict__ pos,
                                const double *__restrict__ par, const int32_t *__restrict__ type,
                                const PairWidths *__restrict__ widths, const int32_t *__restrict__ iface_atom,
                                __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo) {
    const int j = blockIdx.y * blockDim.x + threadIdx.x;
    if (j >= N) return;
    const int u = fmu ? blockIdx.x : blockIdx.x + N;       // wFQ has no dipole rows
    const bool face = u >= N;
    const int i = face ? iface_atom[u - N] : u;
    PairTile t;
    t.qq = 0.0;
    for (int k = 0; k < 3; ++k) t.qm[k] = t.mq[k] = 0.0;
    for (int k = 0; k < 6; ++k) t.mm[k] = 0.0;
    if (i == j) {
        t.qq = par[2 * N + i];
    } else {
        const double dx = pos[i] - pos[j], dy = pos[N + i] - pos[N + j], dz = pos[2 * N + i] - pos[2 * N + j];
        const int ti = type[i], tj = type[j];
        if (fmu) plx_pair_tile_w(dx, dy, dz, widths[ti + nt * tj], ti == tj, t);
        else t.qq = plx_pair_qq_w(dx, dy, dz, widths[ti + nt * tj]);
    }
    auto put = [&](int64_t r, int64_t k, double v) { split_store(v, a_tiled(r, k, ktiles), hi, lo); };
    if (face) {
        const int64_t r = n + (u - N);
        put(r, j, t.qq);
        if (fmu)
            for (int b = 0; b < 3; ++b) put(r, N + 3LL * j + b, t.qm[b]);
        return;
    }
    const int mi[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    for (int a = 0; a < 3; ++a) {
        const int64_t r = N + 3LL * i + a;
        put(r, j, t.mq[a]);
        for (int b = 0; b < 3; ++b) put(r, N + 3LL * j + b, t.mm[mi[a][b]]);
    }
}

// FP64 -> (BF16 high, BF16 low) split of row-major rows [rows][n] into rows of ld
// elements, whose padding stays zero.
__global__ void split_bf16(int rows, int n, const double *__restrict__ in, int64_t ld, __nv_bfloat16 *__restrict__ hi,
                           __nv_bfloat16 *__restrict__ lo) {
    const int64_t total = (int64_t)rows * n;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / n;
        split_store(in[e], r * ld + (e - r * n), hi, lo);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    // initialised once, thread-safely (function-local static)
    static const EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        PLX_CHECK_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        if (!p || q != cudaDriverEntryPointSuccess) throw Error(PLX_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// 2-D BF16 tensor [outer][inner] with leading dimension ld (elements), boxes of
// (kBK inner x box_outer), 64-byte swizzle, zero fill out of bounds.
CUtensorMap make_map(const void *ptr, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_outer) {
    CUtensorMap m;
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {ld * 2};
    cuuint32_t box[2] = {(cuuint32_t)kBK, box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(PLX_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    return m;
}

// Schedule of the launch's tiles on `sms` SMs (one CTA per SM, see TcLaunch): whole
// waves of whole tiles, and the last wave's k-tiles in equal runs -- unless its tiles
// fill at least 0.9 of the chip (splitting would cost more in partial sums than the
// idle SMs) or would be split below kMinRun k-tiles a CTA.  Sets full, run, units and
// the groups' unit0; returns the number of CTAs.
int make_schedule(TcLaunch &L, int sms) {
    const int r = L.tiles % sms;
    L.full = r >= 0.9 * sms ? L.tiles : L.tiles - r;
    L.units = 0;
    for (int g = 0; g < L.ngroups; ++g) {
        TcGroup &gp = L.grp[g];
        const int end = g + 1 < L.ngroups ? L.grp[g + 1].tile0 : L.tiles;
        gp.unit0 = L.units;
        L.units += std::max(0, end - std::max(gp.tile0, L.full)) * gp.ktiles;
    }
    if (L.units == 0) {
        L.run = 1;
        return L.full;
    }
    L.run = std::max(kMinRun, (L.units + sms - 1) / sms);
    return L.full + (L.units + L.run - 1) / L.run;
}

}  // namespace


// The word a launch reports a wait that ran out in; allocated before an operand, which is
// complete once the geometry holds it.
static void error_word(plx_geom *g) {
    if (g->d_tc_err.p) return;
    g->d_tc_err.alloc(g->ctx, 1);
    PLX_CHECK_CUDA(cudaMemsetAsync(g->d_tc_err.p, 0, sizeof(int), g->ctx->stream));
}

// Operands are built in local arrays and handed to the geometry when complete: an
// allocation that the budget refuses half-way leaves the geometry without an operand,
// and a later call builds it again.
void build_t_split(plx_geom *g) {
    if (g->d_Th.p) return;
    if (!g->has_T && is_bem(g)) throw Error(PLX_ERR_ARG, "BEM geometry without its Green-function matrix");
    const int64_t n = g->n_var;
    const int64_t ld = (n + kLdAlign - 1) / kLdAlign * kLdAlign;
    const int64_t rows = (n + kBM - 1) / kBM * kBM, ktiles = ld / kBK;
    g->ldk = ld;
    error_word(g);
    DevArray<uint16_t> Th, Tl;
    Th.alloc(g->ctx, (size_t)(rows * ld));
    Tl.alloc(g->ctx, (size_t)(rows * ld));
    auto *hi = reinterpret_cast<__nv_bfloat16 *>(Th.p);
    auto *lo = reinterpret_cast<__nv_bfloat16 *>(Tl.p);
    if (!g->has_T) {
        // on-the-fly geometry: the split is generated from the pair formulas
        split_tiled_gen<<<dim3((unsigned)ktiles, (unsigned)(rows / kBM)), 256, 0, g->ctx->stream>>>(
            g->n_atoms, (int)n, g->model == PLX_WFQFMU, ktiles, g->d_pos.p, g->d_par.p, hi, lo);
    } else if (g->t_symmetric) {
        split_tiled<<<4096, 256, 0, g->ctx->stream>>>((int)n, ktiles, rows * ld, g->d_T.p, hi, lo);
    } else {
        // stored transposed (BEM): split the transpose
        split_tiled_t<<<dim3((unsigned)ktiles, (unsigned)(rows / kBM)), 256, 0, g->ctx->stream>>>((int)n, ktiles,
                                                                                                 g->d_T.p, hi, lo);
    }
    g->ctx->launches++;
    PLX_CHECK_CUDA(cudaGetLastError());
    g->d_Th.swap(Th);
    g->d_Tl.swap(Tl);
}

// Interface of an alloy: rows I with neighbours of another type, the atoms J
// whose T charge rows the correction needs (I and those neighbours), and the
// cross-type entries of I as a CSR over positions in J.
static void build_interface(plx_geom *g) {
    plx_ctx *ctx = g->ctx;
    cudaStream_t st = ctx->stream;
    const int N = g->n_atoms;
    std::vector<int32_t> rowptr(N + 1), type(N);
    std::vector<int32_t> col((size_t)g->nnz);
    std::vector<double> kt((size_t)g->nnz);
    PLX_CHECK_CUDA(cudaMemcpyAsync(rowptr.data(), g->d_rowptr.p, (N + 1) * 4, cudaMemcpyDeviceToHost, st));
    PLX_CHECK_CUDA(cudaMemcpyAsync(type.data(), g->d_type.p, N * 4, cudaMemcpyDeviceToHost, st));
    if (g->nnz) {
        PLX_CHECK_CUDA(cudaMemcpyAsync(col.data(), g->d_col.p, g->nnz * 4, cudaMemcpyDeviceToHost, st));
        PLX_CHECK_CUDA(cudaMemcpyAsync(kt.data(), g->d_ktval.p, g->nnz * 8, cudaMemcpyDeviceToHost, st));
    }
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));
    std::vector<int32_t> pos(N, -1), J, rows, ptr(1, 0), xcol, xtj;
    std::vector<double> xkt;
    auto place = [&](int a) {
        if (pos[a] < 0) {
            pos[a] = (int32_t)J.size();
            J.push_back(a);
        }
    };
    for (int i = 0; i < N; ++i) {
        bool any = false;
        for (int e = rowptr[i]; e < rowptr[i + 1]; ++e)
            if (type[col[e]] != type[i]) any = true;
        if (!any) continue;
        place(i);
        rows.push_back(i);
        for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) {
            const int j = col[e];
            if (type[j] == type[i]) continue;
            place(j);
            xcol.push_back(j);          // atom index for now
            xtj.push_back(type[j]);
            xkt.push_back(kt[e]);
        }
        ptr.push_back((int32_t)xcol.size());
    }
    for (auto &c : xcol) c = pos[c];
    std::vector<int32_t> ipos(rows.size());
    for (size_t t = 0; t < rows.size(); ++t) ipos[t] = pos[rows[t]];
    g->n_iface = (int)J.size();
    g->n_xrows = (int)rows.size();
    auto up_i = [&](DevArray<int32_t> &d, const std::vector<int32_t> &h) {
        d.alloc(ctx, std::max<size_t>(h.size(), 1));
        if (!h.empty()) PLX_CHECK_CUDA(cudaMemcpyAsync(d.p, h.data(), h.size() * 4, cudaMemcpyHostToDevice, st));
    };
    up_i(g->d_iface_atom, J);
    up_i(g->d_xrow, rows);
    up_i(g->d_xipos, ipos);
    up_i(g->d_xrowptr, ptr);
    up_i(g->d_xcol, xcol);
    up_i(g->d_xtj, xtj);
    g->d_xkt.alloc(ctx, std::max<size_t>(xkt.size(), 1));
    if (!xkt.empty()) PLX_CHECK_CUDA(cudaMemcpyAsync(g->d_xkt.p, xkt.data(), xkt.size() * 8, cudaMemcpyHostToDevice, st));
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));
}

static void build_a_split(plx_geom *g) {
    if (g->d_Ah.p) return;
    const bool hetero = g->n_types > 1;
    if (hetero) build_interface(g);
    const int64_t n = g->n_var;
    const int64_t M = n + (hetero ? g->n_iface : 0);
    const int64_t ld = (n + kLdAlign - 1) / kLdAlign * kLdAlign;
    const int64_t rows = (M + kBM - 1) / kBM * kBM, ktiles = ld / kBK;
    g->ldk = ld;
    g->fold_rows = M;
    error_word(g);
    DevArray<uint16_t> Ah, Al;
    Ah.alloc(g->ctx, (size_t)(rows * ld));
    Al.alloc(g->ctx, (size_t)(rows * ld));
    // rows M..rows of the last m-tile are read by the kernel: zero them
    PLX_CHECK_CUDA(cudaMemsetAsync(Ah.p, 0, (size_t)(rows * ld) * 2, g->ctx->stream));
    PLX_CHECK_CUDA(cudaMemsetAsync(Al.p, 0, (size_t)(rows * ld) * 2, g->ctx->stream));
    const int fmu = g->model == PLX_WFQFMU, N = g->n_atoms;
    auto *hi = reinterpret_cast<__nv_bfloat16 *>(Ah.p);
    auto *lo = reinterpret_cast<__nv_bfloat16 *>(Al.p);
    cudaStream_t st = g->ctx->stream;
    const FoldTarget out{Ah.p, Al.p, ktiles};
    if (M > N && g->has_T) {
        copy_rows_split<<<dim3((unsigned)(M - N), (unsigned)((n + 255) / 256)), 256, 0, st>>>(
            N, (int)n, ktiles, g->d_T.p, g->d_iface_atom.p, hi, lo);
        g->ctx->launches++;
    } else if (M > N) {
        const unsigned units = (unsigned)((fmu ? N : 0) + (M - n));
        pair_rows_split<<<dim3(units, (unsigned)((N + 127) / 128)), 128, 0, st>>>(
            N, (int)n, g->n_types, fmu, ktiles, g->d_pos.p, g->d_par.p, g->d_type.p, g->d_widths.p, g->d_iface_atom.p, hi,
            lo);
        g->ctx->launches++;
    }
    fold_charge_rows(g, out);
    PLX_CHECK_CUDA(cudaGetLastError());
    g->d_Ah.swap(Ah);
    g->d_Al.swap(Al);
}

int64_t tc_fold_rows(plx_geom *g) {
    build_a_split(g);
    return g->fold_rows;
}

void tc_contract_group(const std::vector<TcItem> &items) {
    if (items.empty()) return;
    if ((int)items.size() > kMaxGroups) {
        // more contractions than one launch describes: in launches of kMaxGroups
        for (size_t i0 = 0; i0 < items.size(); i0 += kMaxGroups)
            tc_contract_group(std::vector<TcItem>(items.begin() + i0,
                                                  items.begin() + std::min(items.size(), i0 + kMaxGroups)));
        return;
    }
    plx_ctx *ctx = items[0].g->ctx;
    const int nprod = items[0].nprod;
    for (const TcItem &it : items)
        if (it.g->ctx != ctx || it.nprod != nprod)
            throw Error(PLX_ERR_ARG, "a grouped contraction needs one context and one product count");
    for (size_t i = 0; i < items.size(); ++i)
        for (size_t j = 0; j < i; ++j)
            if (items[i].g == items[j].g) {
                // one geometry twice: its column split buffers hold one operand at a time
                for (const TcItem &it : items) tc_contract_group({it});
                return;
            }
    // longest k first: whole tiles go to the SMs in launch order
    std::vector<int> order(items.size());
    for (size_t i = 0; i < items.size(); ++i) order[i] = (int)i;
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return items[a].g->n_var > items[b].g->n_var; });
    TcLaunch L;
    std::memset(&L, 0, sizeof(L));
    L.ngroups = (int)items.size();
    L.wait_limit = ctx->wait_limit;
    int bn_max = 32;
    const int sms = sm_count(ctx->device);
    for (int k = 0; k < L.ngroups; ++k) {
        const TcItem &it = items[order[k]];
        plx_geom *g = it.g;
        if (it.folded)
            build_a_split(g);
        else
            build_t_split(g);
        const int n = g->n_var;
        // output rows: n, or the folded operand's rows (n plus interface rows); S is [R][M]
        const int M = it.folded ? (int)g->fold_rows : n;
        const int R = 2 * it.count;
        const int64_t ld = g->ldk;
        // column tiles: as few as possible, each a multiple of 16 columns (<= 256, the
        // MMA's N granularity, which keeps the padding of a tile under 16 columns)
        const int ntile = (R + 255) / 256;
        const int bn = ((R + ntile - 1) / ntile + 15) / 16 * 16;
        const int Rpad = ntile * bn;
        if (!it.presplit) {
            tc_column_buffers(g, it.count);
            split_bf16<<<std::min<int64_t>(4096, n_blocks((int64_t)R * n, 256)), 256, 0, ctx->stream>>>(
                R, n, it.X, ld, reinterpret_cast<__nv_bfloat16 *>(g->d_Xh.p),
                reinterpret_cast<__nv_bfloat16 *>(g->d_Xl.p));
            ctx->launches++;
        }
        L.map[k][0] = make_map(g->d_Xh.p, ld, Rpad, ld, bn);
        L.map[k][1] = make_map(g->d_Xl.p, ld, Rpad, ld, bn);
        TcGroup &gp = L.grp[k];
        // A in tile order, one contiguous pre-swizzled 16 KB block per stage tile
        gp.ah = reinterpret_cast<const uint8_t *>(it.folded ? g->d_Ah.p : g->d_Th.p);
        gp.al = reinterpret_cast<const uint8_t *>(it.folded ? g->d_Al.p : g->d_Tl.p);
        gp.M = M;
        gp.R = R;
        gp.bn = bn;
        gp.ktiles = (int)(ld / kBK);
        gp.ctiles = ntile;
        gp.tile0 = L.tiles;
        gp.S = it.S;
        if (it.Y) {
            const bool bem = is_bem(g);
            gp.rows = TcRows{n,
                             bem ? n : g->n_atoms,
                             g->n_types,
                             it.d_freq,
                             bem ? nullptr : g->d_type.p,
                             g->d_dq.p,
                             g->d_frac.p,
                             g->d_inv_alpha.p,
                             it.X,
                             it.Y};
        }
        L.tiles += (M + kBM - 1) / kBM * ntile;
        bn_max = std::max(bn_max, (bn + 31) / 32 * 32);
    }
    // callers poll the words of every geometry of the group
    L.err = items[order[0]].g->d_tc_err.p;
    if (!L.err) throw Error(PLX_ERR_CUDA, "tensor-core error word missing");
    L.bn_max = bn_max;
    const int ctas = make_schedule(L, sms);
    const int split = L.tiles - L.full;
    if (split > 0) {
        plx_geom *g0 = items[order[0]].g;
        const size_t pn = (size_t)(split + ctas - L.full) * kBM * bn_max;
        if (g0->d_tcpart.n < pn) g0->d_tcpart.alloc(ctx, pn);
        L.P = g0->d_tcpart.p;
    }
    L.stages = std::min(8, kSmemBudget / tc_stage_bytes(bn_max, nprod));
    const int smem = L.stages * tc_stage_bytes(bn_max, nprod) + 1024 /* align */ + 256 /* barriers */;
    auto kern = nprod == 1 ? tc_contract_kernel<1> : tc_contract_kernel<3>;
    once_per_device(reinterpret_cast<const void *>(kern), ctx->device, [&] {
        PLX_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    });
    launch_pdl(kern, ctas, kThreadsTc, smem, ctx->stream, L);
    ctx->launches++;
    PLX_CHECK_CUDA(cudaGetLastError());
    if (split > 0) {
        launch_pdl(reduce_pieces, dim3(split, n_blocks(bn_max, kRedCols)), kBM, 0, ctx->stream, L);
        ctx->launches++;
    }
    PLX_CHECK_CUDA(cudaGetLastError());
}

TcColumns tc_column_buffers(plx_geom *g, int count) {
    // rows for every column tiling of up to `count` columns (a tile pads to 16 columns,
    // at most R / 256 + 1 tiles); the padding along k stays zero, rows past the batch
    // feed columns of the product that are not stored
    const size_t rows = 2 * (size_t)count + 16 * ((2 * (size_t)count + 255) / 256);
    const size_t need = rows * g->ldk;
    if (g->d_Xh.n < need) {
        try {
            g->d_Xh.alloc(g->ctx, need);
            g->d_Xl.alloc(g->ctx, need);
        } catch (...) {                      // both or none: the size of one stands for both
            g->d_Xh.release();
            throw;
        }
        PLX_CHECK_CUDA(cudaMemsetAsync(g->d_Xh.p, 0, need * 2, g->ctx->stream));
        PLX_CHECK_CUDA(cudaMemsetAsync(g->d_Xl.p, 0, need * 2, g->ctx->stream));
    }
    return TcColumns{g->d_Xh.p, g->d_Xl.p, g->ldk};
}

TcColumns tc_presplit(plx_geom *g, int count) {
    if (tc_folds_operator(g))
        build_a_split(g);
    else
        build_t_split(g);
    return tc_column_buffers(g, count);
}

void tc_contract(plx_geom *g, int count, const double *X, double *S, int nprod, bool folded) {
    tc_contract_group({TcItem{g, count, X, S, nprod, folded, nullptr, nullptr, false}});
}

int tc_error(plx_geom *g) {
    if (!g->d_tc_err.p) return 0;
    int h = 0;
    PLX_CHECK_CUDA(cudaMemcpyAsync(&h, g->d_tc_err.p, sizeof(int), cudaMemcpyDeviceToHost, g->ctx->stream));
    PLX_CHECK_CUDA(cudaStreamSynchronize(g->ctx->stream));
    // reported once: the next call starts clean
    if (h) PLX_CHECK_CUDA(cudaMemsetAsync(g->d_tc_err.p, 0, sizeof(int), g->ctx->stream));
    return h;
}

}  // namespace plx
