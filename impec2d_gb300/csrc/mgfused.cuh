// Single-CTA coarse V-cycle (included by pressure.cu).
//
// k_coarse_vcycle: the whole V-cycle of the coarse levels (<= 32^2 cells in FP64, <= 64^2 in
// FP32) in one CTA, operators and iterates in shared memory, coarsest level by the dense FP64
// inverse.  Replaces ~10 launches per coarse level.
#pragma once
// Included inside namespace impec of pressure.cu (uses its IX, c_off and Level definitions).

constexpr int MGC_MAXL = 8;

// Coarsest-level solve x = Dinv b in FP64 (n <= 64; for the singular system Dinv, from
// k_dense_invert, is its pseudo-inverse).  Every
// thread of the block takes part (the count of loop trips and shuffles is the same for all):
// row r is summed by the 8 lanes of one lane group, lane g over the columns g, g + 8, g + 16,
// ... in ascending order; an xor butterfly then adds the 8 partials as
// ((p0+p1)+(p2+p3))+((p4+p5)+(p6+p7)) on every lane.  On this FP64 pipe the latency of the
// dependent chain sets the time, so it is kept short: 8 multiply-adds and 3 additions.  The
// coarse V-cycle kernels all solve the coarsest level here, so they give the same bits.
// dinv: row-major, row stride n, in global or shared memory.
template <class T>
__device__ void dense_coarse_apply(int n, const double* dinv, const T* b, T* x) {
    const int t = threadIdx.x, g = t & 7, rows = blockDim.x >> 3;
    for (int base = 0; base < n; base += rows) {
        const int r = base + (t >> 3);
        double s = 0.0;
        if (r < n)
            for (int c = g; c < n; c += 8) s += dinv[r * n + c] * (double)b[c];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        if (r < n && g == 0) x[r] = (T)s;
    }
    __syncthreads();
}

template <class T>
struct CoarseArgs {
    int nl, dn;
    int npre, npost;  // smoother colours before / after the coarse correction
    int post_first;   // five-point: colour of the first one after it
    int zero_color;   // five-point: restriction skips cells of this colour (their residual is ~0), or -1
    int n1[MGC_MAXL], n2[MGC_MAXL];
    const T* tx[MGC_MAXL];
    const T* ty[MGC_MAXL];
    const T* a9[MGC_MAXL];
    const T* id[MGC_MAXL];
    const T* dg[MGC_MAXL];  // diagonals (FACE5; EXP9 uses plane 0 of a9)
    const T* w4[MGC_MAXL];  // transfer weights (FACE5, levels below the first), null: plain transfers
    T* x0;           // iterate of the first handled level (global)
    const T* b0;     // its right-hand side (global)
    const double* dinv;
};

// One colour of a sweep: red-black (0, 1) or four-colour (0..3).
template <class T, int KIND>
__device__ void cv_colour(int n1, int n2, const T* tx, const T* ty, const T* a9, const T* id, const T* b, T* x, int col) {
    const int n = n1 * n2;
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const int i = k / n2, j = k % n2;
        if (KIND == FACE5) {
            if (((i + j) & 1) != col) continue;
            T sm = b[k];
            if (i > 0) sm += tx[IX(i, j, n2)] * x[k - n2];
            if (i < n1 - 1) sm += tx[IX(i + 1, j, n2)] * x[k + n2];
            if (j > 0) sm += ty[IX(i, j, n2 + 1)] * x[k - 1];
            if (j < n2 - 1) sm += ty[IX(i, j + 1, n2 + 1)] * x[k + 1];
            x[k] = sm * id[k];
        } else {  // as k_gs4_exp9: s = b - sum_e a_e x_e, x = s * idiag
            if ((((i & 1) << 1) | (j & 1)) != col) continue;
            T o = 0;
            for (int e = 1; e < 9; ++e) {
                int ii = i + c_off[e][0], jj = j + c_off[e][1];
                if (ii < 0 || ii >= n1 || jj < 0 || jj >= n2) continue;
                o += a9[e * n + k] * x[IX(ii, jj, n2)];
            }
            x[k] = (b[k] - o) * id[k];
        }
    }
    __syncthreads();
}

// Residual sums of the children of coarse cell (I, J) on its east, west, north and south side
// (as k_restrict5; the skipped colour counts as zero).
template <class T>
__device__ __forceinline__ void cv_sides(int I, int J, int n1, int n2, int zc, const T* tx, const T* ty, const T* dg,
                                         const T* b, const T* x, T& e, T& w, T& n, T& s) {
    auto child = [&](int di, int dj) -> T {
        const int i = 2 * I + di, j = 2 * J + dj;
        if (((di + dj) & 1) == zc || i >= n1 || j >= n2) return T(0);
        return resid5<T>(n1, n2, i, j, tx, ty, dg, b, x);
    };
    const T r00 = child(0, 0), r01 = child(0, 1), r10 = child(1, 0), r11 = child(1, 1);
    e = r10 + r11;
    w = r00 + r01;
    n = r01 + r11;
    s = r00 + r10;
}

template <class T, int KIND>
__global__ void __launch_bounds__(1024) k_coarse_vcycle(CoarseArgs<T> A) {
    pdl_enter();
    extern __shared__ __align__(16) unsigned char cv_raw[];
    T* sm = reinterpret_cast<T*>(cv_raw);
    T *tx[MGC_MAXL], *ty[MGC_MAXL], *a9[MGC_MAXL], *id[MGC_MAXL], *dg[MGC_MAXL], *x[MGC_MAXL], *b[MGC_MAXL],
        *w4[MGC_MAXL];
    size_t off = 0;
    for (int l = 0; l < A.nl; ++l) {
        const int n1 = A.n1[l], n2 = A.n2[l], n = n1 * n2;
        tx[l] = ty[l] = a9[l] = dg[l] = w4[l] = nullptr;
        if (KIND == FACE5) {
            tx[l] = sm + off; off += (size_t)(n1 + 1) * n2;
            ty[l] = sm + off; off += (size_t)n1 * (n2 + 1);
            dg[l] = sm + off; off += n;
            if (l > 0 && A.w4[l]) { w4[l] = sm + off; off += (size_t)4 * n; }
        } else {
            a9[l] = sm + off; off += (size_t)9 * n;
        }
        id[l] = sm + off; off += n;
        x[l] = sm + off; off += n;
        b[l] = sm + off; off += n;
    }
    for (int l = 0; l < A.nl; ++l) {
        const int n1 = A.n1[l], n2 = A.n2[l], n = n1 * n2;
        if (KIND == FACE5) {
            for (int k = threadIdx.x; k < (n1 + 1) * n2; k += blockDim.x) stage_async(tx[l] + k, A.tx[l] + k);
            for (int k = threadIdx.x; k < n1 * (n2 + 1); k += blockDim.x) stage_async(ty[l] + k, A.ty[l] + k);
            for (int k = threadIdx.x; k < n; k += blockDim.x) stage_async(dg[l] + k, A.dg[l] + k);
            if (w4[l])
                for (int k = threadIdx.x; k < 4 * n; k += blockDim.x) stage_async(w4[l] + k, A.w4[l] + k);
        } else {
            for (int k = threadIdx.x; k < 9 * n; k += blockDim.x) stage_async(a9[l] + k, A.a9[l] + k);
        }
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            stage_async(id[l] + k, A.id[l] + k);
            if (l == 0) {
                stage_async(x[l] + k, A.x0 + k);
                stage_async(b[l] + k, A.b0 + k);
            } else {
                x[l][k] = T(0);
                b[l][k] = T(0);
            }
        }
    }
    stage_wait();
    __syncthreads();
    const int L = A.nl - 1;  // dense level
    for (int l = 0; l < L; ++l) {
        const int n1 = A.n1[l], n2 = A.n2[l], c1 = A.n1[l + 1], c2 = A.n2[l + 1], nc = c1 * c2;
        for (int s = 0; s < A.npre; ++s)
            cv_colour<T, KIND>(n1, n2, tx[l], ty[l], a9[l], id[l], b[l], x[l], KIND == FACE5 ? s & 1 : s & 3);
        for (int K = threadIdx.x; K < nc; K += blockDim.x) {
            const int I = K / c2, J = K % c2;
            T s = 0;
            if (KIND == FACE5) {  // the neighbours' sides are computed again: few cells, one pass
                auto sides = [&](int I, int J, T& e, T& w, T& n, T& so) {
                    cv_sides<T>(I, J, n1, n2, A.zero_color, tx[l], ty[l], dg[l], b[l], x[l], e, w, n, so);
                };
                const T* w = w4[l + 1];
                T e, we, n, so, d0, d1, d2, d3;
                sides(I, J, e, we, n, so);
                s = e + we;
                if (w) s = restrict_sum<T>(e, we, n, so, w[K], w[nc + K], w[2 * nc + K], w[3 * nc + K]);
                if (w && I > 0) { sides(I - 1, J, d0, d1, d2, d3); s = fma(w[K - c2], d0, s); }
                if (w && I < c1 - 1) { sides(I + 1, J, d0, d1, d2, d3); s = fma(w[nc + K + c2], d1, s); }
                if (w && J > 0) { sides(I, J - 1, d0, d1, d2, d3); s = fma(w[2 * nc + K - 1], d2, s); }
                if (w && J < c2 - 1) { sides(I, J + 1, d0, d1, d2, d3); s = fma(w[3 * nc + K + 1], d3, s); }
            } else {
                for (int a = 0; a < 2; ++a)
                    for (int bb = 0; bb < 2; ++bb) {
                        const int i = 2 * I + a, j = 2 * J + bb;
                        if (i < n1 && j < n2) s += resid9<T>(n1, n2, i, j, a9[l], b[l], x[l]);
                    }
            }
            b[l + 1][K] = s;
            x[l + 1][K] = 0;
        }
        __syncthreads();
    }
    dense_coarse_apply<T>(A.dn, A.dinv, b[L], x[L]);  // coarsest level
    for (int l = L - 1; l >= 0; --l) {
        const int n1 = A.n1[l], n2 = A.n2[l], c1 = A.n1[l + 1], c2 = A.n2[l + 1];
        const T* xc = x[l + 1];
        for (int k = threadIdx.x; k < n1 * n2; k += blockDim.x) {
            const int i = k / n2, j = k % n2;
            x[l][k] = prolong_cell<T>(i, j, n2, x[l], c1, c2, xc, w4[l + 1]);
        }
        __syncthreads();
        for (int s = 0; s < A.npost; ++s)
            cv_colour<T, KIND>(n1, n2, tx[l], ty[l], a9[l], id[l], b[l], x[l],
                               KIND == FACE5 ? (A.post_first + s) & 1 : 3 - (s & 3));
    }
    const int n0 = A.n1[0] * A.n2[0];
    for (int k = threadIdx.x; k < n0; k += blockDim.x) A.x0[k] = x[0][k];
}
