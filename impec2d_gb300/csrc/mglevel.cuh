// Half a V-cycle of one five-point level per launch (included by pressure.cu inside namespace impec).
//
// k_down5: the pre-smoothing from x = 0 (N colours: red, black, red, ...), the residual and the
// restriction; k_up5: the prolongation and the post-smoothing (N colours, in reverse).  A block owns
// a TR x TC tile of the level and keeps it, with a halo, in shared memory: the iterate, b, 1/diag
// and both face planes are read from L2 or HBM once per half cycle, where one launch per colour
// and transfer read them five times.  What a colour on the tile needs of the cells around it is
// computed again in the halo, one ring less for every colour (their values equal what the
// neighbouring tiles compute: same inputs, same arithmetic): 30% more operations on a 16 x 32 tile.
// FP64 is bound by its pipe (1024^2: down 39 us, up 31, at 74 and 85% of it; 43 and 41 us as
// separate launches), FP32 by instruction issue (its large levels take mgmarch.cuh), small levels by the
// number of launches, two instead of eight.
// Per-cell arithmetic and its order are those of k_rb_zero, k_rb_face5, k_restrict5 and
// k_prolong_rb, so the cycle gives the same bits.
//
// Between the two only the colour that the prolongation corrects survives (the other one is
// overwritten unread), so k_down5 writes that colour alone, packed: cell (i, j) at
// i * ((n2 + 1) / 2) + j / 2 of the level's second iterate buffer.  k_up5 writes the first one.  The
// tiles of a launch read no cell that another tile of the launch writes.
#pragma once

constexpr int LV_N = 3, LV_H = 4, LV_T = 256;  // colours per side, halo of the staged tile, threads
template <class T, int TR, int TC>
struct LvTile {
    static constexpr int P = TC + 2 * LV_H, ROWS = TR + 2 * LV_H, PLANE = P * ROWS;  // rows of 16-byte pieces
    static constexpr size_t SMEM = (size_t)5 * PLANE * sizeof(T);  // x, b, 1/diag, tx, ty
    static_assert(TR % 2 == 0 && TC % 8 == 0, "aggregates and 16-byte pieces do not straddle tiles");
};

// Rows [r0, r1) and columns [c0, c1) of the staged tile (which starts at global (i0 - LV_H, j0 - LV_H))
// from a plane with rows of `stride` elements, of which g1 x g2 exist.  vec: 16-byte pieces (the
// plane's rows start on 16-byte boundaries and the piece count is whole; c0 and c1 are widened).
template <class T, int TR, int TC>
__device__ __forceinline__ void lv_stage(T* dst, const T* __restrict__ src, int stride, int g1, int g2, int i0, int j0,
                                         int r0, int r1, int c0, int c1, bool vec) {
    using L = LvTile<T, TR, TC>;
    constexpr int V = 16 / sizeof(T);
    if (vec) {
        const int v0 = c0 / V, nv = (c1 + V - 1) / V - v0;
        for (int k = threadIdx.x; k < (r1 - r0) * nv; k += LV_T) {
            const int r = r0 + k / nv, c = V * (v0 + k % nv), i = i0 - LV_H + r, j = j0 - LV_H + c;
            if (i < 0 || i >= g1 || j < 0 || j >= g2) continue;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst + r * L::P + c)),
                         "l"(src + (size_t)i * stride + j)
                         : "memory");
        }
        return;
    }
    const int nc = c1 - c0;
    for (int k = threadIdx.x; k < (r1 - r0) * nc; k += LV_T) {
        const int r = r0 + k / nc, c = c0 + k % nc, i = i0 - LV_H + r, j = j0 - LV_H + c;
        if (i >= 0 && i < g1 && j >= 0 && j < g2) stage_async(dst + r * L::P + c, src + (size_t)i * stride + j);
    }
}

// The colour `col` on the tile and `ring` rings around it.
template <class T, int TR, int TC, int RING>
__device__ __forceinline__ void lv_colour(T* x, const T* b, const T* id, const T* tx, const T* ty, int n1, int n2, int i0,
                                          int j0, int col, bool zero) {
    constexpr int P = LvTile<T, TR, TC>::P, HC = (TC + 2 * RING) / 2;
    for (int k = threadIdx.x; k < (TR + 2 * RING) * HC; k += LV_T) {
        const int r = LV_H - RING + k / HC, i = i0 - LV_H + r;
        const int c = LV_H - RING + ((i + j0 - RING + col) & 1) + 2 * (k % HC), j = j0 - LV_H + c, o = r * P + c;
        if (i < 0 || i >= n1 || j < 0 || j >= n2) continue;
        T s = b[o];
        if (!zero) {
            if (i > 0) s += tx[o] * x[o - P];
            if (i < n1 - 1) s += tx[o + P] * x[o + P];
            if (j > 0) s += ty[o] * x[o - 1];
            if (j < n2 - 1) s += ty[o + 1] * x[o + 1];
        }
        x[o] = s * id[o];
    }
    __syncthreads();
}

// bc: coarse right-hand side; xc (or null): coarse iterate, set to zero.
template <class T, int TR, int TC>
__global__ void __launch_bounds__(LV_T) k_down5(int n1, int n2, const T* __restrict__ tx, const T* __restrict__ ty,
                                                const T* __restrict__ id, const T* __restrict__ dg,
                                                const T* __restrict__ b, T* __restrict__ xp, int n1c, int n2c,
                                                const T* __restrict__ w4, T* __restrict__ bc, T* __restrict__ xc, int vec) {
    pdl_enter();
    using L = LvTile<T, TR, TC>;
    constexpr int P = L::P;
    extern __shared__ __align__(16) unsigned char lv_raw[];
    T* sx = reinterpret_cast<T*>(lv_raw);
    T *sb = sx + L::PLANE, *sid = sb + L::PLANE, *stx = sid + L::PLANE, *sty = stx + L::PLANE;
    const int i0 = blockIdx.y * TR, j0 = blockIdx.x * TC;
    lv_stage<T, TR, TC>(sb, b, n2, n1, n2, i0, j0, 0, L::ROWS, 0, P, vec);
    lv_stage<T, TR, TC>(sid, id, n2, n1, n2, i0, j0, 0, L::ROWS, 0, P, vec);
    lv_stage<T, TR, TC>(stx, tx, n2, n1 + 1, n2, i0, j0, 1, L::ROWS, 1, P - 1, vec);
    lv_stage<T, TR, TC>(sty, ty, n2 + 1, n1, n2 + 1, i0, j0, 1, L::ROWS - 1, 1, P, false);
    stage_wait();
    __syncthreads();
    lv_colour<T, TR, TC, 4>(sx, sb, sid, stx, sty, n1, n2, i0, j0, 0, true);
    lv_colour<T, TR, TC, 3>(sx, sb, sid, stx, sty, n1, n2, i0, j0, 1, false);
    lv_colour<T, TR, TC, 2>(sx, sb, sid, stx, sty, n1, n2, i0, j0, 0, false);
    // residual of the black cells (the red ones' is zero up to one rounding) on the tile and one
    // ring, in the place of their b; those of the tile also leave their value for k_up5
    constexpr int HC = (TC + 2) / 2;
    const int half = (n2 + 1) / 2;
    for (int k = threadIdx.x; k < (TR + 2) * HC; k += LV_T) {
        const int r = LV_H - 1 + k / HC, i = i0 - LV_H + r;
        const int c = LV_H - 1 + ((i + j0) & 1) + 2 * (k % HC), j = j0 - LV_H + c, o = r * P + c;
        if (i < 0 || i >= n1 || j < 0 || j >= n2) continue;
        T s = sb[o];
        if (i > 0) s += stx[o] * sx[o - P];
        if (i < n1 - 1) s += stx[o + P] * sx[o + P];
        if (j > 0) s += sty[o] * sx[o - 1];
        if (j < n2 - 1) s += sty[o + 1] * sx[o + 1];
        sb[o] = s - dg[IX(i, j, n2)] * sx[o];
        if (r >= LV_H && r < LV_H + TR && c >= LV_H && c < LV_H + TC) xp[(size_t)i * half + (j >> 1)] = sx[o];
    }
    __syncthreads();
    const size_t nc = (size_t)n1c * n2c;
    for (int k = threadIdx.x; k < (TR / 2) * (TC / 2); k += LV_T) {
        const int a = k / (TC / 2), q = k % (TC / 2), I = i0 / 2 + a, J = j0 / 2 + q;
        if (I >= n1c || J >= n2c) continue;
        const int o = (LV_H + 2 * a) * P + LV_H + 2 * q, i = 2 * I, j = 2 * J;
        // the black children: p on the even row (west, north), e on the odd one (east, south)
        auto at = [&](int ii, int jj, int oo) -> T { return ii < n1 && jj < n2 ? sb[oo] : T(0); };
        const T p = at(i, j + 1, o + 1), e = at(i + 1, j, o + P);
        const size_t kk = IX(I, J, n2c);
        T v = restrict_sum<T>(e, p, p, e, w4[kk], w4[nc + kk], w4[2 * nc + kk], w4[3 * nc + kk]);
        if (I > 0) v = fma(w4[kk - n2c], at(i - 1, j, o - P), v);
        if (I < n1c - 1) v = fma(w4[nc + kk + n2c], at(i + 2, j + 1, o + 2 * P + 1), v);
        if (J > 0) v = fma(w4[2 * nc + kk - 1], at(i, j - 1, o - 1), v);
        if (J < n2c - 1) v = fma(w4[3 * nc + kk + 1], at(i + 1, j + 2, o + P + 2), v);
        bc[kk] = v;
        if (xc) xc[kk] = T(0);
    }
}

template <class T, int TR, int TC>
__global__ void __launch_bounds__(LV_T) k_up5(int n1, int n2, const T* __restrict__ tx, const T* __restrict__ ty,
                                              const T* __restrict__ id, const T* __restrict__ b, const T* __restrict__ xp,
                                              T* __restrict__ x, int n1c, int n2c, const T* __restrict__ xc,
                                              const T* __restrict__ w4, const unsigned char* __restrict__ mask, int vec) {
    pdl_enter();
    using L = LvTile<T, TR, TC>;
    constexpr int P = L::P;
    extern __shared__ __align__(16) unsigned char lv_raw[];
    T* sx = reinterpret_cast<T*>(lv_raw);
    T *sb = sx + L::PLANE, *sid = sb + L::PLANE, *stx = sid + L::PLANE, *sty = stx + L::PLANE;
    const int i0 = blockIdx.y * TR, j0 = blockIdx.x * TC;
    lv_stage<T, TR, TC>(sb, b, n2, n1, n2, i0, j0, 2, L::ROWS - 2, 2, P - 2, vec);
    lv_stage<T, TR, TC>(sid, id, n2, n1, n2, i0, j0, 2, L::ROWS - 2, 2, P - 2, vec);
    lv_stage<T, TR, TC>(stx, tx, n2, n1 + 1, n2, i0, j0, 2, L::ROWS - 1, 2, P - 2, vec);
    lv_stage<T, TR, TC>(sty, ty, n2 + 1, n1, n2 + 1, i0, j0, 2, L::ROWS - 2, 2, P - 1, false);
    // corrected black cells on the tile and three rings (the red ones are overwritten unread)
    constexpr int HC = (TC + 6) / 2;
    const int half = (n2 + 1) / 2;
    const size_t nc = (size_t)n1c * n2c;
    for (int k = threadIdx.x; k < (TR + 6) * HC; k += LV_T) {
        const int r = LV_H - 3 + k / HC, i = i0 - LV_H + r;
        const int c = LV_H - 3 + ((i + j0) & 1) + 2 * (k % HC), j = j0 - LV_H + c;
        if (i < 0 || i >= n1 || j < 0 || j >= n2) continue;
        const T old = xp[(size_t)i * half + (j >> 1)];
        T v = old;
        if (!mask || !mask[IX(i, j, n2)]) {  // known cells take no correction
            const int I = i >> 1, J = j >> 1;
            const int I2 = (i & 1) ? min(I + 1, n1c - 1) : max(I - 1, 0), J2 = (j & 1) ? min(J + 1, n2c - 1) : max(J - 1, 0);
            const size_t kk = IX(I, J, n2c);
            v = prolong5<T>(old, xc[kk], xc[IX(I2, J, n2c)], xc[IX(I, J2, n2c)], w4[((i & 1) ? 0 : nc) + kk],
                            w4[((j & 1) ? 2 * nc : 3 * nc) + kk]);
        }
        sx[r * P + c] = v;
    }
    stage_wait();
    __syncthreads();
    lv_colour<T, TR, TC, 2>(sx, sb, sid, stx, sty, n1, n2, i0, j0, 0, false);
    lv_colour<T, TR, TC, 1>(sx, sb, sid, stx, sty, n1, n2, i0, j0, 1, false);
    lv_colour<T, TR, TC, 0>(sx, sb, sid, stx, sty, n1, n2, i0, j0, 0, false);
    for (int k = threadIdx.x; k < TR * TC; k += LV_T) {
        const int r = k / TC, c = k % TC, i = i0 + r, j = j0 + c;
        if (i < n1 && j < n2) x[IX(i, j, n2)] = sx[(r + LV_H) * P + c + LV_H];
    }
}
