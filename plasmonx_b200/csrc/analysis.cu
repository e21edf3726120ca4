// Induced field and plasmon density at points: the analysis step of the
// reference (calculate_induced_field_at_point_{wfq,wfqfmu} and
// calculate_density_at_point_{wfq,wfqfmu}, src/wfq/wfq_module.f90:590-650,
// src/wfq/wfqfmu_module.f90:975-1040, with the kernels
// calculate_induced_field_q / _mu and calculate_density_q / _mu of
// src/matrix/matrix_module.f90:1140-1322).  For d = r_atom - r_point (bohr):
//   E  = E0 e_pol - sum_i q_i d f(r, Rq_i) / r^3                  (r > 0.1)
//      + sum_i [(-3 d d^T / r^5 + I / r^3) fD1 + fD2 d d^T / r^2] mu_i  (r > 0.1)
//   rho = sum_i q_i exp(-r^2/Rq^2) / (pi^3/2 Rq^3)
//       - sum_i 2 exp(-r^2/Rmu^2) / (pi^3/2 Rmu^5) (mu_i . d)
// With fD1, fD2 the damping factors and (mu . d) formed once, an atom's field is
//   d [(-3 fD1 / r^5 + fD2 / r^2) (mu . d) - q f / r^3] + mu fD1 / r^3.
#include <algorithm>
#include <vector>

#include "pair_tiles.cuh"
#include "plx_internal.h"

namespace plx {

namespace {

constexpr int kPts = 128;
constexpr int kProfPoints = 7;   // plx_profile_read category of the point kernels
constexpr double kPi32 = 5.5683279968317078453;   // pi^(3/2)

// Point sums of one launch: the field and density of atoms [a0, a1) at PPT points a
// thread; the atoms are staged through shared memory in tiles, with the reciprocal
// widths and prefactors formed once per atom.
//
// FP64 bound.  A pair takes one rsqrt, one exponential per width and about 50
// operations; the error functions only within seven widths, beyond which the damping
// factors are one in double precision (pair_tiles.cuh), and the exponentials are zero
// beyond 27.3 widths.  Three exponentials, two error functions, a square root and six
// divisions for every pair took 18.4 ms at 1,961 atoms and 64^3 points, now 5.0 ms.
// Two points a thread halve the shared-memory reads of an atom; grids that leave SMs
// idle take one point a thread and split the atoms over blockIdx.y (partial sums
// [y][component][point], added in order by field_reduce): 15^3 points 4,214 -> 131 us, 76,000 points 6,838 -> 1,620 us.
constexpr double kExpZero = 27.3;      // exp(-u^2) is zero in double precision beyond

template <int PPT, bool FMU>
__global__ void __launch_bounds__(kPts) field_points(int N, int achunk, int pol, double e0, int P,
                                                     const double *__restrict__ pos, const double *__restrict__ par,
                                                     const double2 *__restrict__ x, const double *__restrict__ pts,
                                                     double2 *__restrict__ field, double2 *__restrict__ dens,
                                                     double *__restrict__ part) {
    constexpr int NV = FMU ? 15 : 7;
    __shared__ double sa[kPts][NV];    // x, y, z, 1/Rq, density factor, q; 1/Rmu, density and fD2 factors, mu
    double px[PPT], py[PPT], pz[PPT];
    double er[PPT][3], ei[PPT][3], dr[PPT], di[PPT];
#pragma unroll
    for (int u = 0; u < PPT; ++u) {
        const int p = min((int)(blockIdx.x * PPT + u) * kPts + (int)threadIdx.x, P - 1);
        px[u] = pts[p];
        py[u] = pts[P + p];
        pz[u] = pts[2LL * P + p];
        dr[u] = di[u] = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) er[u][k] = ei[u][k] = 0.0;
    }
    const int abeg = blockIdx.y * achunk, aend = min(N, abeg + achunk);
    for (int a0 = abeg; a0 < aend; a0 += kPts) {
        const int a = a0 + threadIdx.x;
        __syncthreads();
        if (a < aend) {
            double *s = sa[threadIdx.x];
            const double rq = par[a];
            const double2 q = x[a];
            s[0] = pos[a];
            s[1] = pos[N + a];
            s[2] = pos[2LL * N + a];
            s[3] = 1.0 / rq;
            s[4] = 1.0 / (kPi32 * rq * rq * rq);
            s[5] = q.x;
            s[6] = q.y;
            if (FMU) {
                const double rm = par[N + a];
                s[7] = 1.0 / rm;
                s[8] = 2.0 / (kPi32 * rm * rm * rm) / (rm * rm);
                for (int k = 0; k < 3; ++k) {
                    const double2 m = x[N + 3LL * a + k];
                    s[9 + 2 * k] = m.x;
                    s[10 + 2 * k] = m.y;
                }
            }
        }
        __syncthreads();
        const int an = min(kPts, aend - a0);
        for (int t = 0; t < an; ++t) {
            const double *s = sa[t];
            const double iq = s[3], gq = s[4], qr = s[5], qi = s[6];
#pragma unroll
            for (int u = 0; u < PPT; ++u) {
                const double d0 = s[0] - px[u], d1 = s[1] - py[u], d2 = s[2] - pz[u];
                const double r2 = d0 * d0 + d1 * d1 + d2 * d2;
                const double ir = rsqrt(r2), r = r2 * ir;
                const bool far = r > 1.0e-1;
                const double ir2 = ir * ir, ir3 = far ? ir2 * ir : 0.0;
                const double uq = r2 == 0.0 ? 0.0 : r * iq;
                const double eq = uq > kExpZero ? 0.0 : exp(-(uq * uq));
                dr[u] = fma(gq * eq, qr, dr[u]);
                di[u] = fma(gq * eq, qi, di[u]);
                double f = ir3;
                if (far && !(uq >= PLX_FAR_WIDTHS)) f = (erf(uq) - (2.0 / PLX_SQRT_PI) * uq * eq) * ir3;
                double tr = -(f * qr), ti = -(f * qi);
                if (FMU) {
                    const double im = s[7];
                    const double um = r2 == 0.0 ? 0.0 : r * im;
                    const double em = um > kExpZero ? 0.0 : exp(-(um * um));
                    const double mdr = s[9] * d0 + s[11] * d1 + s[13] * d2, mdi = s[10] * d0 + s[12] * d1 + s[14] * d2;
                    const double gm = s[8] * em;
                    dr[u] = fma(-gm, mdr, dr[u]);
                    di[u] = fma(-gm, mdi, di[u]);
                    double fd = ir3, fe = 0.0;
                    if (far && !(um >= PLX_FAR_WIDTHS)) {
                        fd = (erf(um) - (2.0 / PLX_SQRT_PI) * um * em) * ir3;
                        fe = (4.0 / PLX_SQRT_PI) * (im * im * im) * em * ir2;
                    }
                    const double A = far ? fma(-3.0 * ir2, fd, fe) : 0.0;
                    tr = fma(A, mdr, tr);
                    ti = fma(A, mdi, ti);
                    er[u][0] = fma(fd, s[9], er[u][0]);
                    ei[u][0] = fma(fd, s[10], ei[u][0]);
                    er[u][1] = fma(fd, s[11], er[u][1]);
                    ei[u][1] = fma(fd, s[12], ei[u][1]);
                    er[u][2] = fma(fd, s[13], er[u][2]);
                    ei[u][2] = fma(fd, s[14], ei[u][2]);
                }
                if (!far) continue;
                er[u][0] = fma(tr, d0, er[u][0]);
                ei[u][0] = fma(ti, d0, ei[u][0]);
                er[u][1] = fma(tr, d1, er[u][1]);
                ei[u][1] = fma(ti, d1, ei[u][1]);
                er[u][2] = fma(tr, d2, er[u][2]);
                ei[u][2] = fma(ti, d2, ei[u][2]);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < PPT; ++u) {
        const int p = (blockIdx.x * PPT + u) * kPts + threadIdx.x;
        if (p >= P) continue;
        if (part) {
            double *o = part + (int64_t)blockIdx.y * 8 * P + p;
            for (int k = 0; k < 3; ++k) {
                o[(int64_t)(2 * k) * P] = er[u][k];
                o[(int64_t)(2 * k + 1) * P] = ei[u][k];
            }
            o[6LL * P] = dr[u];
            o[7LL * P] = di[u];
            continue;
        }
        er[u][pol] += e0;
        if (field)
            for (int k = 0; k < 3; ++k) field[3LL * p + k] = make_double2(er[u][k], ei[u][k]);
        if (dens) dens[p] = make_double2(dr[u], di[u]);
    }
}

__global__ void field_reduce(int P, int ny, int pol, double e0, const double *__restrict__ part,
                             double2 *__restrict__ field, double2 *__restrict__ dens) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;      // k: field component, 3 the density
    if (p >= P) return;
    double re = 0.0, im = 0.0;
    for (int y = 0; y < ny; ++y) {
        const double *o = part + ((int64_t)y * 8 + 2 * k) * P + p;
        re += o[0];
        im += o[P];
    }
    if (k == pol) re += e0;
    if (k < 3) {
        if (field) field[3LL * p + k] = make_double2(re, im);
    } else if (dens) {
        dens[p] = make_double2(re, im);
    }
}

// BEM field at points (calculate_induced_field_at_point_bem,
// src/bem/bem_module.f90:1152-1222, with calculate_induced_field_q_bem,
// src/matrix/matrix_module.f90:1444-1464): the point's first nearest tessera l
// decides inside / outside -- outside when |p - com| > |c_l - com| + 0.5 A,
// com the mean of the centres; inside, the field is zero; outside,
// E = E0 e_pol - sum_i q_i d_i / |d_i|^3 over |d_i| > 0.1 bohr, d_i = c_i - p.
// One thread per point; the centres and charges are read through the cache.
__global__ void __launch_bounds__(kPts) bem_field_points(int n, int P, int pol, double e0, double margin,
                                                         double cx, double cy, double cz,
                                                         const double *__restrict__ c /*[3][n]*/,
                                                         const double2 *__restrict__ q,
                                                         const double *__restrict__ pts /*[3][P]*/,
                                                         double2 *__restrict__ field) {
    const int p = blockIdx.x * kPts + threadIdx.x;
    if (p >= P) return;
    const double px = pts[p], py = pts[P + p], pz = pts[2 * P + p];
    double lowest = 1.0e6;
    int l = 0;
    for (int i = 0; i < n; ++i) {
        const double dx = c[i] - px, dy = c[n + i] - py, dz = c[2 * n + i] - pz;
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        if (lowest > r) {
            lowest = r;
            l = i;
        }
    }
    const double ex = c[l] - cx, ey = c[n + l] - cy, ez = c[2 * n + l] - cz;
    const double gx = px - cx, gy = py - cy, gz = pz - cz;
    double er[3] = {0.0, 0.0, 0.0}, ei[3] = {0.0, 0.0, 0.0};
    if (sqrt(gx * gx + gy * gy + gz * gz) > sqrt(ex * ex + ey * ey + ez * ez) + margin) {
        er[pol] = e0;
        for (int i = 0; i < n; ++i) {
            const double d[3] = {c[i] - px, c[n + i] - py, c[2 * n + i] - pz};
            const double r = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
            if (r > 1.0e-1) {
                const double r3 = r * (r * r);
                const double2 qi = q[i];
                for (int k = 0; k < 3; ++k) {
                    er[k] -= d[k] * qi.x / r3;
                    ei[k] -= d[k] * qi.y / r3;
                }
            }
        }
    }
    for (int k = 0; k < 3; ++k) field[3LL * p + k] = make_double2(er[k], ei[k]);
}

}  // namespace

void bem_field_at_points(plx_ctx *ctx, int n, const double *centres, const double *q, double e0, int pol, int P,
                         const double *points, double *field_out) {
    if (n < 1 || P < 0 || !centres || !q || !points || !field_out)
        throw Error(PLX_ERR_ARG, "BEM field at points: empty surface or null array");
    if (pol < 0 || pol > 2) throw Error(PLX_ERR_ARG, "polarisation index must be 0, 1 or 2");
    if (P == 0) return;
    std::vector<double> c(3 * (size_t)n), pts(3 * (size_t)P);
    double com[3] = {0.0, 0.0, 0.0};
    for (int i = 0; i < n; ++i)
        for (int k = 0; k < 3; ++k) {
            c[(size_t)k * n + i] = centres[3 * (size_t)i + k];
            com[k] += centres[3 * (size_t)i + k] / n;
        }
    for (int i = 0; i < P; ++i)
        for (int k = 0; k < 3; ++k) pts[(size_t)k * P + i] = points[3 * (size_t)i + k];
    cudaStream_t st = ctx->stream;
    DevArray<double> d_c, d_q, d_p, d_f;
    d_c.alloc(ctx, c.size());
    d_q.alloc(ctx, 2 * (size_t)n);
    d_p.alloc(ctx, pts.size());
    d_f.alloc(ctx, 6 * (size_t)P);
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_c.p, c.data(), c.size() * 8, cudaMemcpyHostToDevice, st));
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_q.p, q, 2 * (size_t)n * 8, cudaMemcpyHostToDevice, st));
    PLX_CHECK_CUDA(cudaMemcpyAsync(d_p.p, pts.data(), pts.size() * 8, cudaMemcpyHostToDevice, st));
    const double margin = 0.5 * 1.8897261254578281;   // 0.5 Angstrom in bohr
    prof_begin(ctx);
    bem_field_points<<<n_blocks(P, kPts), kPts, 0, st>>>(n, P, pol, e0, margin, com[0], com[1], com[2], d_c.p,
                                                         reinterpret_cast<const double2 *>(d_q.p), d_p.p,
                                                         reinterpret_cast<double2 *>(d_f.p));
    ctx->launches++;
    PLX_CHECK_CUDA(cudaGetLastError());
    prof_end(ctx, kProfPoints, 0.0, 8.0 * (5.0 * n + 9.0 * P));
    PLX_CHECK_CUDA(cudaMemcpyAsync(field_out, d_f.p, 6 * (size_t)P * 8, cudaMemcpyDeviceToHost, st));
    PLX_CHECK_CUDA(cudaStreamSynchronize(st));
}

void field_at_points(plx_geom *g, int pol, const double *d_x, int P, const double *d_pts, double *d_field,
                     double *d_dens) {
    plx_ctx *ctx = g->ctx;
    prof_begin(ctx);
    const int N = g->n_atoms;
    const bool fmu = g->model == PLX_WFQFMU;
    const auto *x = reinterpret_cast<const double2 *>(d_x);
    auto *fo = reinterpret_cast<double2 *>(d_field), *de = reinterpret_cast<double2 *>(d_dens);
    // Numbers of blocks for a B200 (four and eight an SM); constant, because the parts fix the
    // order of a point's sum and so its bits
    const int pairs = n_blocks(P, 2 * kPts);
    if (pairs >= 592) {
        (fmu ? field_points<2, true> : field_points<2, false>)<<<pairs, kPts, 0, ctx->stream>>>(
            N, N, pol, g->e0, P, g->d_pos.p, g->d_par.p, x, d_pts, fo, de, nullptr);
        ctx->launches++;
    } else {
        // a block for about every resident slot of the chip, at least a tile of atoms each;
        // fewer parts where their sums (up to 10 MB) find no room, one needs none
        const int blocks = n_blocks(P, kPts);
        int ny = std::max(1, std::min(n_blocks(N, kPts), 1184 / blocks)), achunk;
        DevArray<double> part;
        for (;; ny /= 2) {
            achunk = n_blocks(n_blocks(N, ny), kPts) * kPts;
            ny = n_blocks(N, achunk);
            if (ny == 1) break;
            try {
                part.alloc(ctx, 8 * (size_t)P * ny);
                break;
            } catch (const Error &e) {
                if (e.code != PLX_ERR_BUDGET && e.code != PLX_ERR_NOMEM) throw;
            }
        }
        (fmu ? field_points<1, true> : field_points<1, false>)<<<dim3(blocks, ny), kPts, 0, ctx->stream>>>(
            N, achunk, pol, g->e0, P, g->d_pos.p, g->d_par.p, x, d_pts, fo, de, ny > 1 ? part.p : nullptr);
        ctx->launches++;
        if (ny > 1) {
            field_reduce<<<dim3(n_blocks(P, 256), 4), 256, 0, ctx->stream>>>(P, ny, pol, g->e0, part.p, fo, de);
            ctx->launches++;
        }
    }
    PLX_CHECK_CUDA(cudaGetLastError());
    // atoms (positions, widths, the solution) once, points in, field and density out
    prof_end(ctx, kProfPoints, 0.0, 8.0 * (5.0 * g->n_atoms + 2.0 * g->n_var + 3.0 * P + 6.0 * P + 2.0 * P));
}

}  // namespace plx
