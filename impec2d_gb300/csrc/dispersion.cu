// Crank-Nicolson Peaceman dispersion (HyperbolicSolver::DiffusionSplitCN ->
// MGSolver::Solve_Parabolic_cc_to_c, src/MGSolver.cpp:846-1392).
//
// D = phi/|u| (alpha_l u u^T + alpha_t (|u|^2 I - u u^T)) (+ phi Dm I, engine option) at
// x-faces (v from a four-face average) and y-faces (u from a four-face average); alpha is
// the configured value times max(dx,dy).  The nine-point CN matrix (I - dt/2 L) and the
// right-hand side (I + dt/2 L) c are assembled exactly as the reference does (including the
// Neumann folding) and solved by four-colour Gauss-Seidel to the relative residual tol.  With the
// matrix A at hand the right-hand side is 2 c - A c.
//
// Every kernel here is bound by FP64 arithmetic or, where it reads the nine planes (72 B per
// cell), by L2 and HBM.
#include <cmath>

#include "internal.cuh"
#include "reduce.cuh"

namespace impec {

constexpr int DBX = 32, DBY = 8;
#define IX(i, j, n2) ((size_t)(i) * (n2) + (j))
__constant__ int d_off[9][2] = {{0, 0}, {-1, 0}, {-1, -1}, {0, -1}, {1, -1}, {1, 0}, {1, 1}, {0, 1}, {-1, 1}};

struct CNArgs {
    int n1, n2;
    double al, at, dm;        // phi * alpha_l, phi * alpha_t, phi * Dm
    double kxx, kyy, kxy;     // 1 / (2 dx dx), 1 / (2 dy dy), 1 / (8 dx dy)
    double dA;                // dx dy
    int guard;
    int dir_row;   // horizontal source: row N1-2 is Dirichlet, c = 0 (src/MGSolver.cpp:1295-1317, 1361-1367); else -1
};

// Peaceman tensors and the CN matrix in one pass: SetupDiffusionTensorF at x-faces, ...G at y-faces
// (src/MGSolver.cpp:846-919), GetCoefficients_Parabolic (:923-948) with the Neumann folding of
// SetMatrixCoefficients_Parabolic (:997-1321).  dt = scale * dt_dev[0].
// A block owns 32 x 16 cells.  It forms each face's scaled tensor entries once, in shared memory
//   x-face (d11, d12): G = dt / (2 dx dx) d11, H = dt / (8 dx dy) d12;  y-face (d22, d21): likewise,
// (34 / 32 of the faces that the tile needs belong to the next one), and then the nine entries
// of each cell from its four faces: sums of G and H alone.  The scales dt / (..) and the quarter
// of the four-face average go into six factors per block.  About 60 FP64 instructions per cell (17
// of them 1/|u|, 9 the reciprocal of the diagonal) against 80 for separate kernels, which also
// wrote and read 64 B per cell of tensors: 1024^2 198 us before, 133 now.
constexpr int CM_C = 32, CM_R = 16, CM_T = 256;
__global__ void __launch_bounds__(CM_T) k_cn_matrix(CNArgs A, const double* __restrict__ u, const double* __restrict__ v,
                                                    const double* __restrict__ dt_dev, double scale,
                                                    double* __restrict__ a9, double* __restrict__ idiag) {
    pdl_enter();
    __shared__ double su[CM_R + 1][CM_C + 2];  // u at x-faces i0 + r, columns j0 - 1 + q (mirrored)
    __shared__ double sv[CM_R + 2][CM_C + 1];  // v at rows i0 - 1 + r (mirrored), y-faces j0 + q
    __shared__ double gx[CM_R + 1][CM_C], hx[CM_R + 1][CM_C], gy[CM_R][CM_C + 1], hy[CM_R][CM_C + 1];
    __shared__ double f[8];
    const int n1 = A.n1, n2 = A.n2, t = threadIdx.x, i0 = blockIdx.y * CM_R, j0 = blockIdx.x * CM_C;
    if (t == 0) {  // x: al, at / 16, dm, (al - at) / 4 times their scales; y: the same
        const double dt = scale * dt_dev[0], x = dt * A.kxx, y = dt * A.kyy, c = dt * A.kxy * 0.25 * (A.al - A.at);
        f[0] = x * A.al; f[1] = x * A.at * 0.0625; f[2] = x * A.dm; f[3] = c;
        f[4] = y * A.al; f[5] = y * A.at * 0.0625; f[6] = y * A.dm;
    }
    for (int k = t; k < (CM_R + 1) * (CM_C + 2); k += CM_T) {
        const int r = k / (CM_C + 2), q = k % (CM_C + 2), i = min(i0 + r, n1), j = min(max(j0 - 1 + q, 0), n2 - 1);
        su[r][q] = u[IX(i, j, n2)];
    }
    for (int k = t; k < (CM_R + 2) * (CM_C + 1); k += CM_T) {
        const int r = k / (CM_C + 1), q = k % (CM_C + 1), i = min(max(i0 - 1 + r, 0), n1 - 1), j = min(j0 + q, n2);
        sv[r][q] = v[IX(i, j, n2 + 1)];
    }
    __syncthreads();
    // w: the normal velocity, s: four times the tangential one; |.|^2 = w^2 + s^2 / 16
    auto face = [&](double w, double s, double fl, double ft, double fm, double& g, double& h) {
        const double w2 = w * w, s2 = s * s, m = fma(0.0625, s2, w2);
        const double inv = A.guard && m == 0.0 ? 0.0 : rsqrt(m);
        g = fma(inv, fma(ft, s2, fl * w2), fm);
        h = f[3] * inv * (w * s);
    };
    for (int k = t; k < (CM_R + 1) * CM_C; k += CM_T) {
        const int r = k / CM_C, q = k % CM_C;
        face(su[r][q + 1], sv[r][q + 1] + sv[r + 1][q + 1] + sv[r][q] + sv[r + 1][q], f[0], f[1], f[2], gx[r][q], hx[r][q]);
    }
    for (int k = t; k < CM_R * (CM_C + 1); k += CM_T) {
        const int r = k / (CM_C + 1), q = k % (CM_C + 1);
        face(sv[r + 1][q], su[r + 1][q] + su[r + 1][q + 1] + su[r][q] + su[r][q + 1], f[4], f[5], f[6], gy[r][q], hy[r][q]);
    }
    __syncthreads();
    const size_t n = (size_t)n1 * n2;
    for (int k = t; k < CM_R * CM_C; k += CM_T) {
        const int r = k / CM_C, q = k % CM_C, i = i0 + r, j = j0 + q;
        if (i >= n1 || j >= n2) continue;
        const double Gm = gx[r][q], Gp = gx[r + 1][q], Hm = hx[r][q], Hp = hx[r + 1][q];
        const double Km = gy[r][q], Kp = gy[r][q + 1], Jm = hy[r][q], Jp = hy[r][q + 1];
        const double dh = Hm - Hp, dj = Jp - Jm;
        double NW = Hm + Jp, NE = -(Hp + Jp), N = dh - Kp;
        double SW = -(Hm + Jm), SE = Hp + Jm, S = -dh - Km;
        double W = dj - Gm, E = -dj - Gp, C = 1.0 + (Gp + Gm) + (Kp + Km);
        const bool lo = i == 0, hi = i == n1 - 1, le = j == 0, ri = j == n2 - 1;
        if (lo || hi || le || ri) {  // the reference's folding of the entries beyond the edges
            double o[9] = {C, W, SW, S, SE, E, NE, N, NW};
            auto set = [&](double a0, double a1, double a2, double a3, double a4, double a5, double a6, double a7, double a8) {
                o[0] = a0; o[1] = a1; o[2] = a2; o[3] = a3; o[4] = a4; o[5] = a5; o[6] = a6; o[7] = a7; o[8] = a8;
            };
            if (le) set(C + S, W + SW, 0, 0, 0, E + SE, NE, N, NW);
            if (ri) set(C + N, W + NW, SW, S, SE, E + NE, 0, 0, 0);
            if (lo) set(C + W, 0, 0, S + SW, SE, E, NE, N + NW, 0);
            if (hi) set(C + E, W, SW, S + SE, 0, 0, 0, N + NE, NW);
            if (lo && le) set(C + W + S + SW, 0, 0, 0, 0, E + SE, NE, N + NW, 0);
            if (lo && ri) set(C + W + N + NW, 0, 0, S + SW, SE, E + NE, 0, 0, 0);
            if (hi && ri) set(C + N + NE + E, W + NW, SW, S + SE, 0, 0, 0, 0, 0);
            if (hi && le) set(C + S + E + SE, W + SW, 0, 0, 0, 0, 0, N + NE, NW);
            C = o[0]; W = o[1]; SW = o[2]; S = o[3]; SE = o[4]; E = o[5]; NE = o[6]; N = o[7]; NW = o[8];
        }
        if (i == A.dir_row) {
            C = 1. / A.dA;
            W = SW = S = SE = E = NE = N = NW = 0.0;
        }
        double* p = a9 + IX(i, j, n2);
        p[0] = C; p[n] = W; p[2 * n] = SW; p[3 * n] = S; p[4 * n] = SE; p[5 * n] = E; p[6 * n] = NE; p[7 * n] = N; p[8 * n] = NW;
        idiag[IX(i, j, n2)] = 1.0 / C;
    }
}

// x may be written by the kernel that calls this: no read-only loads.
__device__ __forceinline__ double cn_off(int i, int j, int n1, int n2, const double* __restrict__ a9, const double* x) {
    const size_t n = (size_t)n1 * n2, k = IX(i, j, n2);
    double s = 0;
#pragma unroll
    for (int e = 1; e < 9; ++e) {
        int ii = i + d_off[e][0], jj = j + d_off[e][1];
        if (ii < 0 || ii >= n1 || jj < 0 || jj >= n2) continue;
        s += a9[e * n + k] * x[IX(ii, jj, n2)];
    }
    return s;
}

// Right-hand side b = (I + dt/2 L) c = 2 c - A c (SetRHS_Parabolic, src/MGSolver.cpp:1324-1371; 0 on
// known rows), the first iterate, and ||b||^2 into out[0].  The first iterate is the explicit-Euler
// predictor x = 2 b - c = c + dt L c (predict = 0: c): its residual (dt/2 L)(dt L c) is second order in
// dt, against dt/2 L c for c, so one four-colour sweep fewer reaches the tolerance.  Known
// (Dirichlet) rows have b = 0, take x = -c and are exact after the first sweep.  x is not c: the
// neighbours read c.  12 FP64 instructions and 104 B per cell against 25 and two passes for the
// flux form with a separate predictor: 1024^2 59 us before, 31 now.
__global__ void __launch_bounds__(RED_THREADS) k_cn_rhs(int n1, int n2, const double* __restrict__ a9,
                                                        const double* __restrict__ c, double* __restrict__ b,
                                                        double* __restrict__ x, int dir_row, int predict, double* partials,
                                                        int mb, unsigned* counter, double* out) {
    pdl_enter();
    double acc[1] = {0.0};
    for_cells(n1, n2, [&](int i, int j, size_t k) {
        const double cc = c[k];
        double v = fma(2.0 - a9[k], cc, -cn_off(i, j, n1, n2, a9, c));
        if (i == dir_row) v = 0.0;
        b[k] = v;
        x[k] = predict ? fma(2.0, v, -cc) : cc;
        acc[0] += v * v;
    });
    grid_reduce<1>(acc, 0u, partials, mb, counter, out);
}

// Colours of a four-colour Gauss-Seidel sweep on the rows of one parity: the even columns, the odd ones, or
// (both) one after the other.  Rows of one parity do not couple, so a block that takes whole rows
// orders the two colours with its own barrier: two launches per sweep instead of four, and each
// plane's sectors, which hold both column parities, are read once instead of twice (1024^2, a
// sweep: 40 us before, 29 now).  Few long rows make too few blocks for that; there each colour is a launch whose
// blocks share a row (gridDim.y of them; cn_iteration).
constexpr int GS_T = 256;
__global__ void __launch_bounds__(GS_T) k_cn_gs(int n1, int n2, const double* __restrict__ a9,
                                                const double* __restrict__ idiag, const double* __restrict__ b, double* x,
                                                int parity, int first, int last) {
    pdl_enter();
    const int i = 2 * blockIdx.x + parity;
    if (i >= n1) return;
    for (int cj = first; cj <= last; ++cj) {
        if (cj > first) __syncthreads();
        for (int j = 2 * (blockIdx.y * GS_T + threadIdx.x) + cj; j < n2; j += 2 * GS_T * gridDim.y) {
            const size_t k = IX(i, j, n2);
            x[k] = (b[k] - cn_off(i, j, n1, n2, a9, x)) * idiag[k];
        }
    }
}

// ||b - A x||^2 into out[0] after a sweep.  The colour swept last (odd rows and columns) has a
// residual of zero up to one rounding and is left out: a block's segment of an odd row is twice as
// long and takes its even columns only.  1024^2: 38 us before, with ||b||^2, 23 now.
__global__ void __launch_bounds__(RED_THREADS) k_cn_resid(int n1, int n2, const double* __restrict__ a9,
                                                          const double* __restrict__ b, const double* __restrict__ x,
                                                          double* partials, int mb, unsigned* counter, double* out) {
    pdl_enter();
    double acc[1] = {0.0};
    const int even = (n2 + RED_THREADS - 1) / RED_THREADS, odd = ((n2 + 1) / 2 + RED_THREADS - 1) / RED_THREADS;
    const int pair = even + odd, units = (n1 / 2) * pair + (n1 & 1) * even;
    for (int un = blockIdx.x; un < units; un += gridDim.x) {
        const int p = un / pair, s = un - p * pair;
        const int i = 2 * p + (s >= even), j = s < even ? s * RED_THREADS + (int)threadIdx.x
                                                       : 2 * ((s - even) * RED_THREADS + (int)threadIdx.x);
        if (j >= n2) continue;
        const size_t k = IX(i, j, n2);
        const double r = b[k] - fma(a9[k], x[k], cn_off(i, j, n1, n2, a9, x));
        acc[0] += r * r;
    }
    grid_reduce<1>(acc, 0u, partials, mb, counter, out);
}

__global__ void k_cn_check(DevScalars* S, double tol, int max_its, int inc, cudaGraphConditionalHandle h, int use_h) {
    pdl_enter();
    if (inc) { S->cn_cycles++; S->cn_cycles_total++; }
    double bn = S->red[3], rn = S->red[2];
    double rr = bn > 0 ? sqrt(rn / bn) : sqrt(rn);
    S->cn_relres = rr;
    const bool bad = !(rr == rr) || isinf(rr);
    const bool go = !bad && rr > tol && S->cn_cycles < max_its;
    if (bad) S->flags |= FLAG_CN_NAN;
    else if (!go && rr > tol) S->flags |= FLAG_CN_NOT_CONVERGED;
    S->go = go ? 1 : 0;
    if (use_h) cudaGraphSetConditional(h, go ? 1u : 0u);
}

// Peaceman tensors and the CN matrix for the half step dt = scale * dt_dev (launch only).
impec_status cn_setup(impec_ctx* ctx, const double* u, const double* v, double dt_scale, const double* dt_dev) {
    const impec_params& P = ctx->P;
    const Geo& G = ctx->G;
    const double maxdx = G.dx > G.dy ? G.dx : G.dy;
    const CNArgs A{P.N1, P.N2, P.porosity * (P.alpha_l * maxdx), P.porosity * (P.alpha_t * maxdx), P.porosity * P.Dm,
                   1. / (2. * G.dx * G.dx), 1. / (2. * G.dy * G.dy), 1. / (8. * G.dx * G.dy), G.dx * G.dy,
                   P.peaceman_guard, ctx->cn_dir_row};
    ++ctx->nlaunch;
    launch_k(ctx->stream, k_cn_matrix, dim3((P.N2 + CM_C - 1) / CM_C, (P.N1 + CM_R - 1) / CM_R), CM_T, 0, A, u, v, dt_dev,
             dt_scale, ctx->cn_a9, ctx->cn_idiag);
    IMPEC_LAUNCH_CHECK();
    return IMPEC_OK;
}

// Right-hand side from c, first iterate into x (not c), ||b||^2, cycle counter reset (launch only; the
// caller sweeps once before the first check).
impec_status cn_prepare(impec_ctx* ctx, const double* c, double* x) {
    const int n1 = ctx->P.N1, n2 = ctx->P.N2, cap = red_cap(ctx->num_sms, ctx->max_blocks);
    ++ctx->nlaunch;
    launch_k(ctx->stream, k_cn_rhs, seg_blocks(n1, n2, cap), RED_THREADS, 0, n1, n2, (const double*)ctx->cn_a9, c, ctx->cn_b,
             x, ctx->cn_dir_row, ctx->cn_predict, ctx->partials, ctx->max_blocks, ctx->counter, ctx->dscal->red + 3);
    IMPEC_LAUNCH_CHECK();
    IMPEC_CUDA_TRY(cudaMemsetAsync(&ctx->dscal->cn_cycles, 0, sizeof(int), ctx->stream));
    return IMPEC_OK;
}

impec_status cn_check(impec_ctx* ctx, double tol, int inc, cudaGraphConditionalHandle h, int use_h) {
    ++ctx->nlaunch;
    launch_k(ctx->stream, k_cn_check, 1, 1, 0, ctx->dscal, tol, ctx->P.max_cycles, inc, h, use_h);
    IMPEC_LAUNCH_CHECK();
    return IMPEC_OK;
}

// One four-colour Gauss-Seidel sweep (the reference starts from 0, only the iteration count
// differs) followed by the new residual (launch only).
impec_status cn_iteration(impec_ctx* ctx, double* x) {
    const int n1 = ctx->P.N1, n2 = ctx->P.N2, cap = red_cap(ctx->num_sms, ctx->max_blocks);
    const auto colours = [&](int parity, int first, int last, int blocks) {
        ++ctx->nlaunch;
        launch_k(ctx->stream, k_cn_gs, dim3((n1 + 1 - parity) / 2, blocks), GS_T, 0, n1, n2, (const double*)ctx->cn_a9,
                 (const double*)ctx->cn_idiag, (const double*)ctx->cn_b, x, parity, first, last);
    };
    // Rows shared by several blocks where whole rows would leave SMs idle (us of a solve of three sweeps, whole rows /
    // shared: 4 x 65536 1935 / 313, 64 x 16384 1002 / 443, 128 x 8192 673 / 446, 304 x 8192 1166 / 848, 512 x 2048
    // 448 / 437; but 608 x 2048 486 / 493, 1400 x 4096 1776 / 1789, 256 x 1024 230 / 262).
    const bool shared = n2 >= 2048 && n1 <= 4 * ctx->num_sms;
    for (int parity = 0; parity < 2; ++parity) {
        if (shared) {
            for (int cj = 0; cj < 2; ++cj) colours(parity, cj, cj, (n2 + 2 * GS_T - 1) / (2 * GS_T));
        } else {
            colours(parity, 0, 1, 1);
        }
    }
    ++ctx->nlaunch;
    launch_k(ctx->stream, k_cn_resid, seg_blocks(n1, n2, cap), RED_THREADS, 0, n1, n2, (const double*)ctx->cn_a9,
             (const double*)ctx->cn_b, (const double*)x, ctx->partials, ctx->max_blocks, ctx->counter, ctx->dscal->red + 2);
    IMPEC_LAUNCH_CHECK();
    return IMPEC_OK;
}

// Host-driven CN solve of one half step (per-operation entry point).
impec_status dispersion_cn_dev(impec_ctx* ctx, double* c, const double* u, const double* v, double dt_scale,
                               const double* dt_dev, double tol, int* its, double* relres) {
    IMPEC_CUDA_TRY(cudaMemsetAsync(&ctx->dscal->flags, 0, sizeof(int), ctx->stream));
    IMPEC_TRY(cn_setup(ctx, u, v, dt_scale, dt_dev));
    // the first sweep runs before the first check: the predictor's residual is second order
    // in dt but has never been below the tolerance in practice, and a sweep too many from a
    // converged start still leaves a converged iterate
    double* x = ctx->t1;
    IMPEC_TRY(cn_prepare(ctx, c, x));
    IMPEC_TRY(cn_iteration(ctx, x));
    IMPEC_TRY(cn_check(ctx, tol, 1, 0, 0));
    for (;;) {
        IMPEC_TRY(sync_scalars(ctx));
        if (!ctx->hscal->go) break;
        IMPEC_TRY(cn_iteration(ctx, x));
        IMPEC_TRY(cn_check(ctx, tol, 1, 0, 0));
    }
    IMPEC_CUDA_TRY(cudaMemcpyAsync(c, x, (size_t)ctx->P.N1 * ctx->P.N2 * 8, cudaMemcpyDeviceToDevice, ctx->stream));
    if (its) *its = ctx->hscal->cn_cycles;
    if (relres) *relres = ctx->hscal->cn_relres;
    ctx->last_para_its = ctx->hscal->cn_cycles;
    if (ctx->hscal->flags & FLAG_CN_NAN) return IMPEC_ERR_NAN;
    if (ctx->hscal->flags & FLAG_CN_NOT_CONVERGED) return IMPEC_ERR_NOT_CONVERGED;
    return IMPEC_OK;
}

}  // namespace impec
