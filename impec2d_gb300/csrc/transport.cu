// Transport: trapezoidal source integrator and dimensionally split MUSCL / upwind advection.
//
// Ghost cells of the reference (two layers, src/Util.cpp:283-438) are replaced by index
// reflection inside the kernels.  The reference's X sweep also updates the ghost rows
// j < 0, j >= N2 (src/HyperbolicSplitSolver.cpp:128-131); those rows are exact mirror images
// of the updated interior rows (mirrored c and mirrored tangential velocity give the same
// fluxes), so the following Y sweep reads them here by reflecting the interior result.
#include <cmath>
#include <mutex>

#include "internal.cuh"
#include "reduce.cuh"

namespace impec {

constexpr int TBX = 32, TBY = 8;
#define IX(i, j, n2) ((size_t)(i) * (n2) + (j))

// ---------------------------------------------------------------- TR source integrator
// TRIntegrator::Integrate (src/TRIntegrator.cpp:49-71) over the well list (q != 0 cells):
// producers c <- c (1 + dt q/2) / (1 - dt q/2), injectors c <- c + dt c_inj q.
// slot 0/1 receives total_mass_outflux of this call; S->total_outflux += |tmo|.
__global__ void __launch_bounds__(RED_THREADS) k_tr(int nw, const int* __restrict__ idx, const double* __restrict__ qv,
                                                    double* __restrict__ c, const double* __restrict__ dt_dev,
                                                    double scale, double cinj, DevScalars* S, int slot) {
    pdl_enter();
    const double dt = scale * dt_dev[0];
    double acc[1] = {0.0};
    for (int w = threadIdx.x; w < nw; w += blockDim.x) {
        const int k = idx[w];
        const double qij = qv[w];
        if (qij < 0) {
            double m = c[k];
            double cn = c[k] * (1 + 0.5 * dt * qij) / (1 - 0.5 * dt * qij);
            c[k] = cn;
            acc[0] += cn - m;
        } else if (qij > 0) {
            c[k] += dt * cinj * qij;
        }
    }
    block_reduce<1>(acc, 0u);
    if (threadIdx.x == 0) {
        if (slot == 0) S->tmo_pre = acc[0]; else S->tmo_post = acc[0];
        S->total_outflux += fabs(acc[0]);
    }
}

impec_status tr_integrate_dev(impec_ctx* ctx, double* c, double dt_scale, const double* dt_dev, int slot) {
    if (!ctx->have_source || ctx->nwells == 0) return IMPEC_OK;
    ++ctx->nlaunch, launch_k(ctx->stream, k_tr, 1, RED_THREADS, 0, ctx->nwells, ctx->well_idx, ctx->well_q, c, dt_dev, dt_scale,
                                             ctx->P.inj_fluid_conc, ctx->dscal, slot);
    IMPEC_LAUNCH_CHECK();
    return IMPEC_OK;
}

// ---------------------------------------------------------------- limiter and upwind selection
// Comparisons on the integer pipe.  FP64 compares issue on the FP64 pipe, the bottleneck of
// the transport kernels on GB300; for non-NaN doubles these are exact equivalents (a NaN
// operand still yields a NaN result through the arithmetic around them).
// x > 0: the bit pattern, read as a signed integer, is positive (+0 is 0, negatives are < 0).
__device__ __forceinline__ bool pos(double x) { return __double_as_longlong(x) > 0LL; }
// The reference limiter xi(r) = min(2r/(1+r), 2/(1+r)) times (a+b)/2 (src/MUSCLSplitSolver.cpp:54-93)
// equals, in exact arithmetic, minmod(a, b): r = a/b <= 1 gives a, r > 1 gives b, opposite signs give 0.
// IEEE magnitudes order like their bit patterns with the sign bit cleared.  The halves are masked
// and compared as 32-bit words: a 64-bit mask of the sign bit is compiled to an FP64 absolute
// value, one more FP64 instruction per slope (1024^2, X then Y: 29 instead of 26 per cell).
__device__ __forceinline__ double minmod(double a, double b) {
    const int ha = __double2hiint(a), hb = __double2hiint(b), la = __double2loint(a), lb = __double2loint(b);
    const unsigned ua = ha & 0x7fffffff, ub = hb & 0x7fffffff;
    const bool opposite = (ha ^ hb) < 0, le = ua < ub || (ua == ub && (unsigned)la <= (unsigned)lb);
    return __hiloint2double(opposite ? 0 : le ? ha : hb, opposite ? 0 : le ? la : lb);
}

// WAF intercell flux times dt / (dx phi) (hyper_method "waf_split" / "waf"; the reference parses
// these, src/SimParams.cpp:200-208, but ships no source for them).  Toro's weighted average flux
// with the van Leer limiter (Riemann Solvers and Numerical Methods for Fluid Dynamics, 3rd ed., ch.
// 13-14): cr is the face's Courant number, A = 1 - (1 - |cr|) * 2r / (1 + r) for r > 0 (else 1, the
// upwind flux), r = upwind jump / local jump, F = cr ((1 + s A) cL + (1 - s A) cR) / 2, s = sign(cr).
__device__ __forceinline__ double waf_face(double cr, double cLL, double cL, double cR, double cRR) {
    const double dloc = cR - cL;
    double A = 1.0;
    if (dloc != 0.0) {
        const double dupw = cr >= 0.0 ? cL - cLL : cRR - cR;
        const double r = dupw / dloc;
        if (r > 0.0) A = 1.0 - (1.0 - fabs(cr)) * (2.0 * r / (1.0 + r));
    }
    const double s = cr > 0.0 ? 1.0 : (cr < 0.0 ? -1.0 : 0.0);
    return 0.5 * (1.0 + s * A) * (cr * cL) + 0.5 * (1.0 - s * A) * (cr * cR);
}

// Reflected (or wrapped) cell index, clamped into [0, n): tile loads may reach further than
// two cells past the boundary on small grids; those values never reach an in-domain output.
template <int BC>
__device__ __forceinline__ int cell_at(int i, int n) {
    int r = BC == IMPEC_BC_PERIODIC ? wrap_cell(i, n) : refl_cell(i, n);
    return r < 0 ? 0 : (r >= n ? n - 1 : r);
}

// Normal face velocity along the sweep direction, ghost faces by odd reflection (Neumann)
// or wrap-around (periodic).
template <int BC>
__device__ __forceinline__ double face_at(const double* __restrict__ u, int f, int n, size_t stride_f, size_t off) {
    if (BC == IMPEC_BC_PERIODIC) {
        int w = wrap_face(f, n);
        w = w < 0 ? 0 : (w > n ? n : w);
        return u[(size_t)w * stride_f + off];
    }
    double s = 1.0;
    int ff = refl_face(f, n, s);
    ff = ff < 0 ? 0 : (ff > n ? n : ff);
    return s * u[(size_t)ff * stride_f + off];
}

// ---------------------------------------------------------------- split sweeps cell by cell
// For grids too small to fill the GPU with tiles (below): a thread per cell forms everything its
// cell needs, more operations than a tile's strips but one short chain per launch.
//
// Cell reconstruction and Hancock half step (src/MUSCLSplitSolver.cpp:54-93, :121-129).
// kap = 0.5 dt / (dx phi).  sl: state at the cell's left face, sr: at its right face.
__device__ __forceinline__ void hancock(double cm, double c0, double cp, double ul, double ur, double kap,
                                        double& sl, double& sr) {
    const double d = minmod(c0 - cm, cp - c0);
    const double UR = fma(0.5, d, c0), UL = fma(-0.5, d, c0);
    const double df = kap * (ul * UL - ur * UR);
    sl = UL + df;
    sr = UR + df;
}

// One sweep along a line: cells k in [0,n) at positions base + k*cs of c, faces f in [0,n]
// at base_f + f*fs of the face array.  Computes the update of cell k.
// cg (may be null) supplies the cells outside [0,n) instead of the reflection of c.
template <int SCHEME, int BC>
__device__ __forceinline__ double sweep_cell(const double* __restrict__ c, const double* __restrict__ cg,
                                             size_t cbase, size_t cs, const double* __restrict__ u, size_t ubase,
                                             size_t us, int k, int n, double kap, double lam) {
    auto C = [&](int m) {
        const double* src = (cg && (m < 0 || m >= n)) ? cg : c;
        return src[cbase + (size_t)cell_at<BC>(m, n) * cs];
    };
    auto U = [&](int f) { return face_at<BC>(u, f, n, us, ubase); };
    double uw = U(k), ue = U(k + 1);
    double Fw, Fe;
    if (SCHEME == IMPEC_UPWINDSPLIT) {  // src/UpwindSplitSolver.cpp:43-65
        double cm = C(k - 1), c0 = C(k), cp = C(k + 1);
        Fw = uw * (pos(uw) ? cm : c0);
        Fe = ue * (pos(ue) ? c0 : cp);
        return c0 + lam * (Fw - Fe);
    }
    if (SCHEME == IMPEC_WAFSPLIT) {
        double cmm = C(k - 2), cm = C(k - 1), c0 = C(k), cp = C(k + 1), cpp = C(k + 2);
        return c0 + (waf_face(uw * lam, cmm, cm, c0, cp) - waf_face(ue * lam, cm, c0, cp, cpp));
    }
    double cmm = C(k - 2), cm = C(k - 1), c0 = C(k), cp = C(k + 1), cpp = C(k + 2);
    double uww = U(k - 1), uee = U(k + 2);
    double slm, srm, sl0, sr0, slp, srp;
    hancock(cmm, cm, c0, uww, uw, kap, slm, srm);
    hancock(cm, c0, cp, uw, ue, kap, sl0, sr0);
    hancock(c0, cp, cpp, ue, uee, kap, slp, srp);
    (void)slm;
    (void)srp;
    Fw = uw * (pos(uw) ? srm : sl0);
    Fe = ue * (pos(ue) ? sr0 : slp);
    return c0 + lam * (Fw - Fe);
}

// X sweep: lines along i (stride N2), faces u (N1+1) x N2.
template <int SCHEME, int BC>
__global__ void k_sweep_x(int n1, int n2, const double* __restrict__ cin, const double* __restrict__ cghost,
                          double* __restrict__ cout, const double* __restrict__ u, const double* __restrict__ dt_dev,
                          double dt_scale, double inv_dx_phi) {
    pdl_enter();
    int j = blockIdx.x * TBX + threadIdx.x, i = blockIdx.y * TBY + threadIdx.y;
    if (i >= n1 || j >= n2) return;
    const double dt = dt_scale * dt_dev[0];
    const double lam = dt * inv_dx_phi, kap = 0.5 * lam;
    cout[IX(i, j, n2)] = sweep_cell<SCHEME, BC>(cin, cghost, j, n2, u, j, n2, i, n1, kap, lam);
}

// Y sweep: lines along j (stride 1), faces v N1 x (N2+1).
template <int SCHEME, int BC>
__global__ void k_sweep_y(int n1, int n2, const double* __restrict__ cin, double* __restrict__ cout,
                          const double* __restrict__ v, const double* __restrict__ dt_dev, double dt_scale,
                          double inv_dy_phi) {
    pdl_enter();
    int j = blockIdx.x * TBX + threadIdx.x, i = blockIdx.y * TBY + threadIdx.y;
    if (i >= n1 || j >= n2) return;
    const double dt = dt_scale * dt_dev[0];
    const double lam = dt * inv_dy_phi, kap = 0.5 * lam;
    cout[IX(i, j, n2)] = sweep_cell<SCHEME, BC>(cin, nullptr, IX(i, 0, n2), 1, v, IX(i, 0, n2 + 1), 1, j, n2, kap, lam);
}

// ---------------------------------------------------------------- split sweeps on a tile
// The dimensionally split update (src/HyperbolicSplitSolver.cpp:51-159) of one TI x TJ tile: X, Y,
// Y after X, X after Y, or (symmetric-parallel) the average of the last two.  All of them are
// FP64-bound on GB300 (1.06 TFLOP/s), so the arithmetic is arranged for the fewest operations.
//
// With W = dt u / (dx phi) at the faces, the MUSCL-Hancock sweep (src/MUSCLSplitSolver.cpp:54-189)
//   L, R = c -+ d/2 + (W_w (c - d/2) - W_e (c + d/2)) / 2,   c' = c + W_w s_w - W_e s_e,
// s the upwind cell's state at the face (R of the cell before it where W > 0, else L of the cell
// after it), is evaluated as
//   base = E c,  E = 1 + (W_w - W_e) / 2;   s = base_up + d_up F,  F = (1/2 - S/4) or -(1/2 + S/4),
// S = W_w + W_e of the upwind cell.  E (per cell) and F (per face) hold no c: the two sweeps that a
// symmetric update makes in each direction share them.  A thread takes a strip of four cells along
// the sweep, so that slopes, bases and face states are computed once (plus the strip's ends): 6.5
// operations per cell and sweep, 43 per cell of a symmetric update with the halo, against 72
// when every cell formed both of its states and both of its fluxes.  1024^2, symmetric MUSCL:
// 152 us before, 95 now (84% of the FP64 pipe); a call with X then Y 160 -> 80 us, Strang 308 -> 118.
//
// The tile: an SM's FP64 units belong to its four sub-partitions (one warp instruction in 64
// cycles each), so a block's warps should fill them evenly.  32 x 32 with strips of four gives 18
// warps for the first sweeps and 16 for the second ones; strips of eight need fewer operations (39)
// but come as 9 and 8 warps, which leaves sub-partitions idle (125 against 109 us a call), as do
// 16 x 32 (118) and 28 x 28 with strips of seven (118).
//
// Shared memory (pitch 37: rows fall into different banks, so a warp can take one strip each of
// 32 rows or of 32 columns): c with its two-cell halo, W, E and F of both directions, and the
// results of the first sweeps (X(c) in the place of c); 85 KB, two blocks per SM.  The first
// sweep covers the cells that the second one reads: 36 lines instead of 32.
constexpr int TJ = 32, STRIP = 4, TP = (TJ + 4) | 1;
enum { MODE_SYM = 0, MODE_XY = 1, MODE_YX = 2, MODE_X = 3, MODE_Y = 4 };  // XY: X, then Y on its result
template <int TI, int MODE>
struct Tile {
    static constexpr int X1 = (TJ + 4) * (TI / STRIP), Y1 = (TI + 4) * (TJ / STRIP);  // strips of a first sweep
    static constexpr int X2 = TJ * (TI / STRIP), Y2 = TI * (TJ / STRIP);              // strips of a second one
    static constexpr int STRIPS = MODE == MODE_SYM  ? X1 + Y1
                                  : MODE == MODE_XY ? (X1 > Y2 ? X1 : Y2)
                                  : MODE == MODE_YX ? (Y1 > X2 ? Y1 : X2)
                                  : MODE == MODE_X  ? X1
                                                    : Y1;
    static constexpr int THREADS = (STRIPS + 31) / 32 * 32;  // the strips of the largest phase, in whole warps
    // planes of shared memory: c, three per direction, Y(c) beside X(c)
    static constexpr int PLANE = (TI + 4) * TP;
    static constexpr size_t SMEM = sizeof(double) * PLANE * (MODE == MODE_SYM ? 8 : MODE == MODE_X || MODE == MODE_Y ? 4 : 7);
};

struct TileArgs {
    int n1, n2;
    const double* cin;
    const double* cghost;  // cells beyond the x ends are taken from here (null: from cin)
    double* cout;
    const double* u;
    const double* v;
    const double* dt;      // device scalar
    double fx, fy;         // scale / (dx phi), scale / (dy phi)
    int row0;              // tile row of block row b: b == 0 ? 0 : row0 + b
};

// One strip: out[k] = new value of cell k (cells at c + k cs, faces at W + k ws, E at e + k cs', F as W).
// c[-2 .. STRIP + 1], W[0 .. STRIP], E[-1 .. STRIP], F[0 .. STRIP] are read.
template <int SCHEME>
__device__ __forceinline__ void sweep_strip(const double* c, int cs, const double* W, const double* E, const double* F,
                                            int ws, double (&out)[STRIP]) {
    if (SCHEME == IMPEC_WAFSPLIT) {
        double cll = c[-2 * cs], cl = c[-cs], c0 = c[0], t = 0.0;
#pragma unroll
        for (int m = 0; m <= STRIP; ++m) {
            const double cr = c[(m + 1) * cs], f = waf_face(W[m * ws], cll, cl, c0, cr);
            if (m > 0) out[m - 1] = t - f;
            t = c0 + f;
            cll = cl; cl = c0; c0 = cr;
        }
        return;
    }
    if (SCHEME == IMPEC_UPWINDSPLIT) {  // src/UpwindSplitSolver.cpp:43-65
        double cl = c[-cs], t = 0.0;
#pragma unroll
        for (int m = 0; m <= STRIP; ++m) {
            const double c0 = c[m * cs], w = W[m * ws], s = pos(w) ? cl : c0;
            if (m > 0) out[m - 1] = fma(-w, s, t);
            t = fma(w, s, c0);
            cl = c0;
        }
        return;
    }
    double c0 = c[-cs], a = c0 - c[-2 * cs], d1 = 0.0, b1 = 0.0, t = 0.0;
#pragma unroll
    for (int m = -1; m <= STRIP; ++m) {
        const double cr = c[(m + 1) * cs], an = cr - c0;
        const double d = minmod(a, an), b = E[m * ws] * c0;
        if (m >= 0) {
            const double w = W[m * ws];
            const bool p = pos(w);
            const double s = fma(p ? d1 : d, F[m * ws], p ? b1 : b);
            if (m > 0) out[m - 1] = fma(-w, s, t);
            t = fma(w, s, c0);
        }
        c0 = cr; a = an; d1 = d; b1 = b;
    }
}

template <int SCHEME, int BC, int MODE, int TI>
__global__ void __launch_bounds__(Tile<TI, MODE>::THREADS) k_advect_tile(const TileArgs A) {
    pdl_enter();
    using L = Tile<TI, MODE>;
    constexpr int NT = L::THREADS, PL = L::PLANE, X1 = L::X1, Y1 = L::Y1, X2 = L::X2, Y2 = L::Y2;
    constexpr bool XF = MODE == MODE_SYM || MODE == MODE_XY || MODE == MODE_X;  // a first sweep in x
    constexpr bool YF = MODE == MODE_SYM || MODE == MODE_YX || MODE == MODE_Y;
    constexpr bool HASX = MODE != MODE_Y, HASY = MODE != MODE_X;
    extern __shared__ double adv_sm[];
    double* sc = adv_sm;                  // c: rows i0-2 .., columns j0-2 ..; then X(c) over it
    double* wx = sc + PL;                 // W of x-faces i0-1 .. (rows), columns as c
    double* ex = wx + (HASX ? PL : 0);    // E of cells i0-1 .. (rows)
    double* fx = ex + (HASX ? PL : 0);    // F of x-faces i0 .. at row f - i0 + 1 (as wx)
    double* wy = fx + (HASX ? PL : 0);    // W of y-faces j0-1 .. (columns), rows as c
    double* ey = wy + (HASY ? PL : 0);    // E of cells j0-1 .. (columns)
    double* fy = ey + (HASY ? PL : 0);    // F of y-faces j0 .. at column f - j0 + 1 (as wy)
    double* s1 = sc;                      // X(c): rows i0 .. at row i - i0 + 2, columns as c
    double* s2 = MODE == MODE_SYM ? fy + PL : sc;  // Y(c): rows as c, columns j0 .. at column j - j0 + 2
    const int n1 = A.n1, n2 = A.n2, t = threadIdx.x;
    const int ti = blockIdx.y == 0 ? 0 : A.row0 + (int)blockIdx.y;
    const int i0 = ti * TI, j0 = blockIdx.x * TJ;
    const double dt = A.dt[0], lx = dt * A.fx, ly = dt * A.fy;
    // ---- c and W (reflected or wrapped ghosts; tiles off the edges need none) ----
    const bool inside = i0 >= 2 && j0 >= 2 && i0 + TI + 2 <= n1 && j0 + TJ + 2 <= n2;
    for (int k = t; k < (TI + 4) * (TJ + 4); k += NT) {
        const int a = k / (TJ + 4), b = k % (TJ + 4), i = i0 - 2 + a, j = j0 - 2 + b, o = a * TP + b;
        if (inside) {
            const size_t g = IX(i, j, n2);
            sc[o] = A.cin[g];
            if (HASX && a < TI + 3) wx[o] = lx * A.u[g + n2];                       // face i + 1
            if (HASY && b < TJ + 3) wy[o] = ly * A.v[IX(i, j + 1, n2 + 1)];         // face j + 1
        } else {
            const int ic = cell_at<BC>(i, n1), jc = cell_at<BC>(j, n2);
            const double* src = A.cghost && (i < 0 || i >= n1) ? A.cghost : A.cin;
            sc[o] = src[IX(ic, jc, n2)];
            if (HASX && a < TI + 3) wx[o] = lx * face_at<BC>(A.u, i + 1, n1, n2, jc);
            if (HASY && b < TJ + 3) wy[o] = ly * face_at<BC>(A.v + IX(ic, 0, n2 + 1), j + 1, n2, 1, 0);
        }
    }
    __syncthreads();
    // ---- E and F ----
    if (SCHEME == IMPEC_MUSCL) {
        for (int k = t; k < (TI + 4) * (TJ + 4); k += NT) {
            const int a = k / (TJ + 4), b = k % (TJ + 4), o = a * TP + b;
            if (HASX && a < TI + 2) {  // cell i0-1+a between wx rows a, a+1; the face above it is wx row a+1
                const double w = wx[o], e = wx[o + TP];
                ex[o] = fma(0.5, w - e, 1.0);
                if (a < TI + 1) {
                    const bool p = pos(e);  // operands are selected, not results: one sum, one multiply-add
                    fx[o + TP] = fma(-0.25, e + (p ? w : wx[o + 2 * TP]), p ? 0.5 : -0.5);
                }
            }
            if (HASY && b < TJ + 2) {
                const double w = wy[o], e = wy[o + 1];
                ey[o] = fma(0.5, w - e, 1.0);
                if (b < TJ + 1) {
                    const bool p = pos(e);
                    fy[o + 1] = fma(-0.25, e + (p ? w : wy[o + 2]), p ? 0.5 : -0.5);
                }
            }
        }
        __syncthreads();
    }
    // ---- first sweeps: X(c) on all columns, Y(c) on all rows; the results wait in registers
    // until every strip has read c, which X(c) then replaces ----
    double r[STRIP];
    const bool xs = XF && t < X1, ys = YF && t >= (XF ? X1 : 0) && t < (XF ? X1 : 0) + Y1;
    const int q = XF ? t - X1 : t;
    const int xb = t % (TJ + 4), xm = STRIP * (t / (TJ + 4)), ya = q % (TI + 4), ym = STRIP * (q / (TI + 4));
    if (xs)
        sweep_strip<SCHEME>(sc + (xm + 2) * TP + xb, TP, wx + (xm + 1) * TP + xb, ex + (xm + 1) * TP + xb,
                            fx + (xm + 1) * TP + xb, TP, r);
    if (ys)
        sweep_strip<SCHEME>(sc + ya * TP + ym + 2, 1, wy + ya * TP + ym + 1, ey + ya * TP + ym + 1, fy + ya * TP + ym + 1, 1,
                            r);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < STRIP; ++k) {
        if (xs) s1[(xm + 2 + k) * TP + xb] = r[k];
        if (ys) s2[ya * TP + ym + 2 + k] = r[k];
    }
    __syncthreads();
    // ---- second sweeps: Y on X(c) and X on Y(c) ----
    const int p = MODE == MODE_SYM ? t - Y2 : t;
    const bool y2 = (MODE == MODE_SYM || MODE == MODE_XY) && t < Y2, x2 = (MODE == MODE_SYM || MODE == MODE_YX) && p >= 0 && p < X2;
    const int ay = 2 + t % TI, my = STRIP * (t / TI), bx = 2 + p % TJ, mx = STRIP * (p / TJ);
    if (y2)
        sweep_strip<SCHEME>(s1 + ay * TP + my + 2, 1, wy + ay * TP + my + 1, ey + ay * TP + my + 1, fy + ay * TP + my + 1, 1,
                            r);
    if (x2)
        sweep_strip<SCHEME>(s2 + (mx + 2) * TP + bx, TP, wx + (mx + 1) * TP + bx, ex + (mx + 1) * TP + bx,
                            fx + (mx + 1) * TP + bx, TP, r);
    if (MODE == MODE_SYM || MODE == MODE_XY || MODE == MODE_YX) __syncthreads();
    if (MODE == MODE_SYM) {  // the threads that hold X(Y(c)) average and write: one column each
        if (y2) {
#pragma unroll
            for (int k = 0; k < STRIP; ++k) s1[ay * TP + my + 2 + k] = r[k];
        }
        __syncthreads();
        if (x2) {
            const int j = j0 + bx - 2;
#pragma unroll
            for (int k = 0; k < STRIP; ++k) {
                const int i = i0 + mx + k;
                if (i < n1 && j < n2) A.cout[IX(i, j, n2)] = 0.5 * (s1[(mx + 2 + k) * TP + bx] + r[k]);
            }
        }
        return;
    }
    if (MODE == MODE_XY || MODE == MODE_YX) {
#pragma unroll
        for (int k = 0; k < STRIP; ++k) {
            if (y2) sc[ay * TP + my + 2 + k] = r[k];
            if (x2) sc[(mx + 2 + k) * TP + bx] = r[k];
        }
        __syncthreads();
    }
    for (int k = t; k < TI * TJ; k += NT) {
        const int a = k / TJ, b = k % TJ, i = i0 + a, j = j0 + b;
        if (i < n1 && j < n2) A.cout[IX(i, j, n2)] = sc[(a + 2) * TP + b + 2];
    }
}

// Launches one tile kernel, whose shared memory is above the default limit.
template <int SCHEME, int BC, int MODE, int TI>
static cudaError_t launch_tile(cudaStream_t s, TileArgs A, bool edges) {
    int rows = (A.n1 + TI - 1) / TI;
    if (edges && rows > 3) {  // tile rows 0, rows - 2, rows - 1 (the last may hold one row only)
        A.row0 = rows - 3;
        rows = 3;
    }
    const cudaError_t e = allow_smem<k_advect_tile<SCHEME, BC, MODE, TI>>((int)Tile<TI, MODE>::SMEM);
    if (e != cudaSuccess) return e;
    const dim3 g((A.n2 + TJ - 1) / TJ, rows);
    return launch_k(s, k_advect_tile<SCHEME, BC, MODE, TI>, g, Tile<TI, MODE>::THREADS, Tile<TI, MODE>::SMEM, A);
}

// Tiles of 8 rows instead of 32: where those of 32 would leave SMs without one (symmetric MUSCL, us of a
// call, 8 / 32 rows: 256^2 36 / 38, 400 x 300 42 / 38, for more of the first sweeps is halo), and where
// their last rows would be a quarter or more of the grid's tiles beyond it (8 x 16384 42 / 75, 16 x 16384 54 / 75,
// 33 x 4096 46 / 50, 48 x 4096 50 / 50; WAF 102 / 225, 158 / 258, 121 / 142, 138 / 142; but 96 x 4096 69 / 64).
static bool tiles_of_8(int n1, int n2) {
    const int rows8 = (n1 + 7) / 8 * 8, rows32 = (n1 + 31) / 32 * 32;
    return (size_t)n1 * n2 < 98304 || 3 * (long)rows32 >= 4 * (long)rows8;
}

template <int SCHEME, int MODE>
static cudaError_t launch_tile_bc(int bc, cudaStream_t s, const TileArgs& A, bool edges) {
    const bool small = tiles_of_8(A.n1, A.n2);
    if (bc == IMPEC_BC_PERIODIC)
        return small ? launch_tile<SCHEME, IMPEC_BC_PERIODIC, MODE, 8>(s, A, edges)
                     : launch_tile<SCHEME, IMPEC_BC_PERIODIC, MODE, 32>(s, A, edges);
    return small ? launch_tile<SCHEME, IMPEC_BC_NEUMANN, MODE, 8>(s, A, edges)
                 : launch_tile<SCHEME, IMPEC_BC_NEUMANN, MODE, 32>(s, A, edges);
}

// hmtype: IMPEC_MUSCL, IMPEC_WAFSPLIT / IMPEC_WAF, else upwind.  edges: only the tile rows that
// hold the two rows next to each x end.
template <int MODE>
static cudaError_t launch_tiles(int hmtype, int bc, cudaStream_t s, const TileArgs& A, bool edges = false) {
    if (hmtype == IMPEC_MUSCL) return launch_tile_bc<IMPEC_MUSCL, MODE>(bc, s, A, edges);
    if (hmtype == IMPEC_WAFSPLIT || hmtype == IMPEC_WAF) return launch_tile_bc<IMPEC_WAFSPLIT, MODE>(bc, s, A, edges);
    return launch_tile_bc<IMPEC_UPWINDSPLIT, MODE>(bc, s, A, edges);
}

// ---------------------------------------------------------------- corner transport upwind
// hyper_method "ctu" (parsed by the reference, src/SimParams.cpp:200-208, no source shipped):
// Colella's unsplit second-order CTU (J. Comput. Phys. 87 (1990) 171-200) on face velocities.
// Each face takes its upwind cell's value extrapolated to the face and the half time level --
// the central slope (unlimited, the recorded order is "2nd order"), the normal Courant
// correction, and half the transverse upwind advection of that cell -- and the interior is
// updated conservatively in one pass.  lx = dt/(dx phi), ly = dt/(dy phi) per unit velocity.
template <int BC>
__global__ void k_ctu(int n1, int n2, const double* __restrict__ cin, double* __restrict__ cout,
                      const double* __restrict__ u, const double* __restrict__ v, const double* __restrict__ dt_dev,
                      double inv_dx_phi, double inv_dy_phi) {
    pdl_enter();
    const int j = blockIdx.x * TBX + threadIdx.x, i = blockIdx.y * TBY + threadIdx.y;
    if (i >= n1 || j >= n2) return;
    const double dt = dt_dev[0], lx = dt * inv_dx_phi, ly = dt * inv_dy_phi;
    auto C = [&](int a, int b) { return cin[IX(cell_at<BC>(a, n1), cell_at<BC>(b, n2), n2)]; };
    // x-face f of row b (normal: odd reflection across x walls; row b: even reflection)
    auto U = [&](int f, int b) { return face_at<BC>(u, f, n1, n2, cell_at<BC>(b, n2)); };
    // y-face f of row a
    auto V = [&](int a, int f) { return face_at<BC>(v + IX(cell_at<BC>(a, n1), 0, n2 + 1), f, n2, 1, 0); };
    auto ty = [&](int a, int b) {  // cell-centred v times its upwind y difference, cell (a, b)
        const double bc = 0.5 * (V(a, b) + V(a, b + 1));
        return bc * (bc >= 0.0 ? C(a, b) - C(a, b - 1) : C(a, b + 1) - C(a, b));
    };
    auto tx = [&](int a, int b) {
        const double ac = 0.5 * (U(a, b) + U(a + 1, b));
        return ac * (ac >= 0.0 ? C(a, b) - C(a - 1, b) : C(a + 1, b) - C(a, b));
    };
    auto Fx = [&](int f) {  // x-face f of row j
        const double vel = U(f, j);
        const int m = vel >= 0.0 ? f - 1 : f;
        const double sx = 0.5 * (C(m + 1, j) - C(m - 1, j));
        const double st = vel >= 0.0 ? C(m, j) + 0.5 * (1.0 - vel * lx) * sx - 0.5 * ly * ty(m, j)
                                     : C(m, j) - 0.5 * (1.0 + vel * lx) * sx - 0.5 * ly * ty(m, j);
        return vel * st;
    };
    auto Fy = [&](int f) {  // y-face f of row i
        const double vel = V(i, f);
        const int m = vel >= 0.0 ? f - 1 : f;
        const double sy = 0.5 * (C(i, m + 1) - C(i, m - 1));
        const double st = vel >= 0.0 ? C(i, m) + 0.5 * (1.0 - vel * ly) * sy - 0.5 * lx * tx(i, m)
                                     : C(i, m) - 0.5 * (1.0 + vel * ly) * sy - 0.5 * lx * tx(i, m);
        return vel * st;
    };
    cout[IX(i, j, n2)] = C(i, j) + lx * (Fx(i) - Fx(i + 1)) + ly * (Fy(j) - Fy(j + 1));
}

static dim3 tgrid(int n1, int n2) { return dim3((n2 + TBX - 1) / TBX, (n1 + TBY - 1) / TBY); }

// One launch of a tile mode on the context's grid; x and y sweeps over x_scale dt and y_scale dt.
template <int MODE>
static impec_status advect_tiles(impec_ctx* ctx, const double* cin, double* cout, const double* u, const double* v,
                                 double x_scale, double y_scale, const double* dt_dev, const double* cghost = nullptr,
                                 bool edges = false) {
    const impec_params& P = ctx->P;
    const TileArgs A{P.N1, P.N2, cin, cghost, cout, u, v, dt_dev, x_scale / (ctx->G.dx * P.porosity),
                     y_scale / (ctx->G.dy * P.porosity), 0};
    ++ctx->nlaunch;
    IMPEC_CUDA_TRY(launch_tiles<MODE>(P.hmtype, P.bc, ctx->stream, A, edges));
    return IMPEC_OK;
}

// The cell-by-cell sweeps.
static impec_status sweep_cells(impec_ctx* ctx, bool x, const double* cin, double* cout, const double* vel, double dt_scale,
                                const double* dt_dev, const double* cghost = nullptr) {
    const impec_params& P = ctx->P;
    const dim3 g = tgrid(P.N1, P.N2), b(TBX, TBY);
    const double f = 1.0 / ((x ? ctx->G.dx : ctx->G.dy) * P.porosity);
    auto go = [&](auto kx, auto ky) {
        return x ? launch_k(ctx->stream, kx, g, b, 0, P.N1, P.N2, cin, cghost, cout, vel, dt_dev, dt_scale, f)
                 : launch_k(ctx->stream, ky, g, b, 0, P.N1, P.N2, cin, cout, vel, dt_dev, dt_scale, f);
    };
    const bool per = P.bc == IMPEC_BC_PERIODIC;
    ++ctx->nlaunch;
#define IMPEC_SWEEP(S)                                                                                       \
    (per ? go(k_sweep_x<S, IMPEC_BC_PERIODIC>, k_sweep_y<S, IMPEC_BC_PERIODIC>)                              \
         : go(k_sweep_x<S, IMPEC_BC_NEUMANN>, k_sweep_y<S, IMPEC_BC_NEUMANN>))
    if (P.hmtype == IMPEC_MUSCL) IMPEC_CUDA_TRY(IMPEC_SWEEP(IMPEC_MUSCL));
    else if (P.hmtype == IMPEC_WAFSPLIT || P.hmtype == IMPEC_WAF) IMPEC_CUDA_TRY(IMPEC_SWEEP(IMPEC_WAFSPLIT));
    else IMPEC_CUDA_TRY(IMPEC_SWEEP(IMPEC_UPWINDSPLIT));
#undef IMPEC_SWEEP
    return IMPEC_OK;
}

// Whether sweeps in a row run cell by cell (microseconds a call, cells / tiles): below 2^16 cells
// tiles do not fill the GPU and their phases take longer than two short launches (180^2, X then Y:
// 22 / 27; Strang 35 / 41; 256^2: 27 / 27, 43 / 42; 512^2: 48 / 38, 82 / 58).  Upwind sweeps have so
// little to compute that the tile's copy back costs more than the second launch up to 2^20 cells
// (512^2: 24 / 26; 1024^2: 42 / 39), in Strang's three tile launches up to 2^18 (360^2: 33 / 34;
// 512^2: 37 / 36).  Rows of the last tiles that lie beyond the grid count against tiles (33 x 2000, WAF:
// 49 / 53); grids of five or fewer rows always go cell by cell (4 x 65536: 53 / 64, Strang 93 / 106, WAF
// 105 / 140 and 188 / 302).
static bool by_cells(const impec_params& P) {
    const size_t n = (size_t)P.N1 * P.N2, rows8 = (size_t)(P.N1 + 7) / 8 * 8;
    const bool upwind = P.hmtype != IMPEC_MUSCL && P.hmtype != IMPEC_WAFSPLIT && P.hmtype != IMPEC_WAF;
    return 2 * rows8 > 3 * (size_t)P.N1 || n * P.N1 < rows8 << (!upwind ? 16 : P.dim_splitting == IMPEC_STRANG ? 18 : 20);
}
// A single sweep: also wherever its tiles would be of 8 rows (33 x 4096, X: 32 / 31, WAF 46 / 52; 256^2 28 / 29, 34 / 37).
static bool sweep_by_cells(const impec_params& P) { return by_cells(P) || tiles_of_8(P.N1, P.N2); }

impec_status advect_x_dev(impec_ctx* ctx, const double* cin, double* cout, const double* u, double dt_scale,
                          const double* dt_dev) {
    if (sweep_by_cells(ctx->P)) return sweep_cells(ctx, true, cin, cout, u, dt_scale, dt_dev);
    return advect_tiles<MODE_X>(ctx, cin, cout, u, nullptr, dt_scale, 0.0, dt_dev);
}

impec_status advect_y_dev(impec_ctx* ctx, const double* cin, double* cout, const double* v, double dt_scale,
                          const double* dt_dev) {
    if (sweep_by_cells(ctx->P)) return sweep_cells(ctx, false, cin, cout, v, dt_scale, dt_dev);
    return advect_tiles<MODE_Y>(ctx, cin, cout, nullptr, v, 0.0, dt_scale, dt_dev);
}

// AdvectSplit (src/HyperbolicSplitSolver.cpp:51-106), cin -> cout; pfs 0 = X_SWEEP, 1 = Y_SWEEP.  cout may
// be cin; if not, cin's values are lost.  s1, s2, s3: scratch fields, none of them cin or cout.
impec_status advect_split_dev(impec_ctx* ctx, double* cin, double* cout, double* s1, double* s2, double* s3, const double* u,
                              const double* v, const double* dt_dev, int* pfs) {
    const impec_params& P = ctx->P;
    const size_t bytes = (size_t)P.N1 * P.N2 * 8;
    // one-launch updates read neighbouring tiles' old values: in place they go through s1
    double* to = cout == cin ? s1 : cout;
    auto back = [&]() -> impec_status {
        if (to != cout) IMPEC_CUDA_TRY(cudaMemcpyAsync(cout, to, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
        return IMPEC_OK;
    };
    if (P.hmtype == IMPEC_CTU) {  // unsplit: one CTU update; the alternating-sweep state stays as it was
        const double fx = 1.0 / (ctx->G.dx * P.porosity), fy = 1.0 / (ctx->G.dy * P.porosity);
        const auto k = P.bc == IMPEC_BC_PERIODIC ? k_ctu<IMPEC_BC_PERIODIC> : k_ctu<IMPEC_BC_NEUMANN>;
        ++ctx->nlaunch;
        launch_k(ctx->stream, k, tgrid(P.N1, P.N2), dim3(TBX, TBY), 0, P.N1, P.N2, (const double*)cin, to, u, v, dt_dev, fx, fy);
        IMPEC_LAUNCH_CHECK();
        return back();
    }
    bool x_first = true;
    switch (P.dim_splitting) {
        case IMPEC_ALTERNATING: x_first = *pfs == 1; break;
        case IMPEC_X_FIRST: break;
        case IMPEC_Y_FIRST: x_first = false; break;
        case IMPEC_STRANG:
            // Advect_X leaves the ghost columns i < 0, i >= N1 untouched, so after X(dt/2), Y(dt)
            // they hold Y(dt) applied to the mirrored input, not mirrors of the new interior; the
            // last X(dt/2) reads them there (src/HyperbolicSplitSolver.cpp:80-85, :128-131, :152-155).
            // Only the two rows next to each end are ever read, so with tiles Y(dt) of the input runs
            // there only.
            *pfs = 0;
            if (by_cells(P)) {
                double* mid = cout == cin ? s3 : cin;  // the input is done with after two sweeps
                IMPEC_TRY(sweep_cells(ctx, false, cin, s2, v, 1.0, dt_dev));
                IMPEC_TRY(sweep_cells(ctx, true, cin, s1, u, 0.5, dt_dev));
                IMPEC_TRY(sweep_cells(ctx, false, s1, mid, v, 1.0, dt_dev));
                return sweep_cells(ctx, true, mid, cout, u, 0.5, dt_dev, s2);
            }
            IMPEC_TRY(advect_tiles<MODE_Y>(ctx, cin, s2, nullptr, v, 0.0, 1.0, dt_dev, nullptr, true));
            IMPEC_TRY(advect_tiles<MODE_XY>(ctx, cin, s1, u, v, 0.5, 1.0, dt_dev));
            return advect_tiles<MODE_X>(ctx, s1, cout, u, nullptr, 0.5, 0.0, dt_dev, s2);
        default:
            *pfs = 0;
            IMPEC_TRY(advect_tiles<MODE_SYM>(ctx, cin, to, u, v, 1.0, 1.0, dt_dev));
            return back();
    }
    *pfs = x_first ? 0 : 1;
    if (by_cells(P)) {  // two launches through s1, no copy
        IMPEC_TRY(sweep_cells(ctx, x_first, cin, s1, x_first ? u : v, 1.0, dt_dev));
        return sweep_cells(ctx, !x_first, s1, cout, x_first ? v : u, 1.0, dt_dev);
    }
    IMPEC_TRY(x_first ? advect_tiles<MODE_XY>(ctx, cin, to, u, v, 1.0, 1.0, dt_dev)
                      : advect_tiles<MODE_YX>(ctx, cin, to, u, v, 1.0, 1.0, dt_dev));
    return back();
}

}  // namespace impec

// ---------------------------------------------------------------- allocation-free transport step
// For callers that cannot allocate device memory: code running under a host framework that
// owns every device allocation (a fixed memory pool or budget), or a caller that must not
// trigger cudaMalloc's implicit device synchronisation in the middle of its own work.  The
// symmetric-parallel update above needs one field-sized buffer (it cannot update c in place,
// since neighbouring tiles read the old c) and a device copy of dt; here both live in a
// file-scope device array that every GPU loading this library holds until the process exits.
// Nothing in the array has to start at zero: each call writes dt and every cell of the
// updated field before any kernel reads them.
namespace impec {

constexpr size_t NOALLOC_MAX_CELLS = size_t(1) << 20;  // 1,048,576 cells: 8 MiB of FP64
constexpr size_t NOALLOC_FIELD_OFFSET = 32;            // doubles before the field (dt at [0]); 256-byte aligned
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_FIELD_OFFSET + NOALLOC_MAX_CELLS];

// Stores dt in the scratch.  dt travels as a kernel argument, so the value itself is what a
// launch (or a captured launch node) carries; a host-to-device copy would instead carry the
// address of the caller's stack variable.
__global__ void k_noalloc_store_dt(double* __restrict__ dst, double dt) { dst[0] = dt; }

// Device address of g_noalloc_scratch on the current device, looked up once per device (the
// host-side name of the array is only a stand-in, not a device address).  The address is kept
// for the life of the process: after cudaDeviceReset on that device this entry point must not
// be called again.
static impec_status noalloc_scratch(double** out) {
    static std::mutex mu;
    static double* addr[64] = {nullptr};
    int dev = 0;
    IMPEC_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) { set_error("device ordinal out of range"); return IMPEC_ERR_ARG; }
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void* p = nullptr;
        IMPEC_CUDA_TRY(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        addr[dev] = static_cast<double*>(p);
    }
    *out = addr[dev];
    return IMPEC_OK;
}

}  // namespace impec

extern "C" impec_status impec_advect_symmetric_noalloc(const impec_params* P, double* c_dev, const double* u_dev,
                                                       const double* v_dev, double dt, void* stream) {
    using namespace impec;
    if (!P || !c_dev || !u_dev || !v_dev) { set_error("null argument"); return IMPEC_ERR_ARG; }
    if (P->N1 < 2 || P->N2 < 2) { set_error("N1 and N2 must be >= 2"); return IMPEC_ERR_ARG; }
    if ((size_t)P->N1 * (size_t)P->N2 > NOALLOC_MAX_CELLS) {
        set_error("impec_advect_symmetric_noalloc: N1*N2 exceeds its static scratch of 1048576 cells; "
                  "use impec_advect_split with a context instead");
        return IMPEC_ERR_ARG;
    }
    if (P->hmtype != IMPEC_MUSCL && P->hmtype != IMPEC_UPWINDSPLIT) { set_error("unknown hmtype"); return IMPEC_ERR_ARG; }
    if (P->bc != IMPEC_BC_NEUMANN && P->bc != IMPEC_BC_PERIODIC) { set_error("unknown bc"); return IMPEC_ERR_ARG; }
    if (P->dim_splitting != IMPEC_SYMMETRIC_PARALLEL) {
        set_error("impec_advect_symmetric_noalloc performs only the symmetric-parallel splitting; "
                  "set dim_splitting to IMPEC_SYMMETRIC_PARALLEL");
        return IMPEC_ERR_ARG;
    }
    if (!(P->porosity > 0) || !(P->x_ub > P->x_lb) || !(P->y_ub > P->y_lb) || !(dt >= 0) || isinf(dt)) {
        set_error("invalid porosity, domain or dt");
        return IMPEC_ERR_ARG;
    }
    double* scratch = nullptr;
    IMPEC_TRY(noalloc_scratch(&scratch));
    cudaStream_t s = (cudaStream_t)stream;
    const int N1 = P->N1, N2 = P->N2;
    const double dx = (P->x_ub - P->x_lb) / N1, dy = (P->y_ub - P->y_lb) / N2;
    const double fx = 1.0 / (dx * P->porosity), fy = 1.0 / (dy * P->porosity);
    double* cnew = scratch + NOALLOC_FIELD_OFFSET;
    launch_k(s, k_noalloc_store_dt, 1, 1, 0, scratch, dt);
    const TileArgs A{N1, N2, c_dev, nullptr, cnew, u_dev, v_dev, scratch, fx, fy, 0};
    IMPEC_CUDA_TRY(launch_tiles<MODE_SYM>(P->hmtype, P->bc, s, A));
    IMPEC_LAUNCH_CHECK();
    IMPEC_CUDA_TRY(cudaMemcpyAsync(c_dev, cnew, (size_t)N1 * N2 * sizeof(double), cudaMemcpyDeviceToDevice, s));
    return IMPEC_OK;
}
