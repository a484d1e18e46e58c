// Cluster V-cycle (included by pressure.cu inside namespace impec).
//
// The coarse levels of one V-cycle (<= 128^2 cells by default) in a single launch of one
// thread-block cluster of up to 16 CTAs.  Each CTA keeps a band of rows of every level in its
// shared memory: for five-point operators the faces, 1/diagonal, diagonal, iterate, right-hand
// side, transfer weights and child residuals; for nine-point ones the nine coefficient planes,
// 1/diagonal, iterate and right-hand side, smoothed by four-colour Gauss-Seidel (the arithmetic of
// k_gs4_exp9).  The phases of the cycle (one colour of a sweep, the two halves of the restriction,
// the prolongation) are separated by cluster barriers.  The smallest levels (<= 256 cells by
// default) and the dense coarsest solve run on CTA 0 alone, with block barriers.  Each cell is
// updated with the arithmetic of the per-level kernels (k_rb_face5, k_restrict5, k_prolong, the
// dense solve of k_coarse_vcycle) in the same order, so the cycle gives the same bits as those
// launches.
//
// Row ownership: level l's rows are cut into bands of rows[l] rows (an even number, so a 2x2
// restriction aggregate never straddles two CTAs); CTA r owns rows [r*rows[l], (r+1)*rows[l]).
// Levels nd .. nl-1 have rows[l] = n1[l]: CTA 0 owns all of them.
//
// What bounds it: latency.  A phase is one dependent chain of 5 to 10 FP64 operations per cell
// (at 128^2 also 1,300 cycles of FP64 issue per colour on 16 SMs) behind a barrier: some forty phases, 26 of them
// behind a cluster barrier at 128^2, the others on CTA 0 alone.  So a five-point band keeps the neighbours' edge rows in halo rows of its own, which the
// neighbour writes when it updates its edge cell (the store's way to the other SM overlaps the
// rest of the phase) instead of being read from there at the start of the next one, and cells are
// found without an integer division.
//
// Staging: every CTA copies its bands (and CTA 0 the coarsest inverse) with asynchronous
// element copies (cp.async), all in flight at once, and waits for them once.  That takes 11,000 of
// the launch's 100,000 cycles, so the kernel is launched with programmatic serialisation: it stages
// its operators while the kernel before it, the restriction that produces its right-hand side,
// still runs (300 x 130 solve 1.80 -> 1.71 ms, 1024^2 step 4.20 -> 4.16, alternating runs).  A solve
// whose finest level is the cluster's has no such kernel in front inside its loop.
// Members of an ensemble launch it without: the waiting clusters keep 16 SMs each from the other members (64
// members of 128^2, a step: 9.14 ms with, 7.69 without).
//
// Measured without gain (100,000 instead of 101,000 cycles): each thread's cell and its
// coefficients held in registers over a level's colours.  A colour of a small level then takes 650
// cycles instead of 1,000, but fetching them takes as long, and the rest is the barrier (1,000 to
// 1,400 cycles, 26 of them), the gathers and the prolongations.
//
// Every barrier is reached by all threads of all CTAs the same number of times (the counts
// depend only on the arguments), and no CTA touches another's shared memory after the last one.
#pragma once
// Needs <cooperative_groups.h>, included at the top of pressure.cu.

constexpr int CL_MAXL = 10;
constexpr int CL_THREADS = 512;
constexpr int CL_MAX_CTAS = 16;
// shared arrays of a level.  Five-point: X, P, Q, P2, Q2 and the four planes of W have a halo row above and
// below the band (plane stride (rows + 2) * n2); plain transfers have no W, and only a restriction that
// takes both colours has P2, Q2.  A nine-point level keeps its nine planes at CL_TX (plane stride rows * n2) and has
// no CL_TY / CL_DG (the diagonal is plane 0), no halo rows and none of the last five.
enum { CL_TX = 0, CL_TY, CL_ID, CL_DG, CL_X, CL_B, CL_W, CL_P, CL_Q, CL_P2, CL_Q2, CL_ARRAYS };

template <class T>
struct ClusterArgs {
    int nl;    // levels handled: 0 .. nl-1 (nl-1 is the dense coarsest level)
    int nd;  // levels 0 .. nd-1 are spread over the cluster; nd .. nl-1 live on CTA 0
    int dn;
    int npre, npost;  // smoother colours before / after the coarse correction
    int post_first;   // five-point: colour of the first one after it
    int zero_color;   // five-point: restriction skips cells of this colour (their residual is ~0), -1: none
    int zero0;        // five-point: level 0 starts from x = 0 (x0 is not read)
    int plain;        // five-point: transfers without weights (as k_restrict5 and prolong_cell without w4)
    int n1[CL_MAXL], n2[CL_MAXL], rows[CL_MAXL];
    float rhalf[CL_MAXL], rn2[CL_MAXL];       // 1 / ((n2 + 1) / 2), 1 / n2
    unsigned off[CL_MAXL][CL_ARRAYS];  // shared-memory offsets (elements of T)
    const T* tx[CL_MAXL];
    const T* ty[CL_MAXL];
    const T* id[CL_MAXL];
    const T* dg[CL_MAXL];
    const T* w4[CL_MAXL];
    const T* a9[CL_MAXL];  // nine-point planes (EXP9)
    T* x0;        // iterate of level 0 (global), read at the start (unless zero0) and written at the end
    const T* b0;  // right-hand side of level 0 (global)
    const double* dinv;
    unsigned dinv_off;  // byte offset in shared memory of CTA 0's copy of dinv
};

// Pointer to row i of array `arr` of level l, in the shared memory of the CTA that owns it.
template <class T>
__device__ __forceinline__ T* cl_row(const cooperative_groups::cluster_group& cl, T* sm, int rank,
                                     const ClusterArgs<T>& A, int l, int arr, int i, int stride) {
    const int R = A.rows[l];
    const int o = i / R;
    T* p = sm + A.off[l][arr] + (size_t)(i - o * R) * stride;
    return o == rank ? p : cl.map_shared_rank(p, (unsigned)o);
}

// Band of level l owned by `rank`: rows [lo, lo + cnt).
template <class T>
__device__ __forceinline__ void cl_band(const ClusterArgs<T>& A, int l, int rank, int& lo, int& cnt) {
    lo = rank * A.rows[l];
    const int hi = lo + A.rows[l] < A.n1[l] ? lo + A.rows[l] : A.n1[l];
    cnt = hi > lo ? hi - lo : 0;
}

// k / n for 0 <= k < 2^16 and n <= 2^15, rn = 1.0f / n: k + 1/2 lies at least 1/2 away from the
// multiples of n, far more than the rounding of the product.
__device__ __forceinline__ int cl_div(int k, float rn) { return (int)(((float)k + 0.5f) * rn); }

// ---- five-point levels
// The rows of the neighbouring CTAs' halos that this band's first and last row go to (X, P or Q of
// level l); null where there is no neighbour.
template <class T>
__device__ __forceinline__ void cl_halo(const cooperative_groups::cluster_group& cl, T* sm, int rank,
                                        const ClusterArgs<T>& A, int l, int arr, int lo, int cnt, T*& up, T*& dn) {
    up = dn = nullptr;
    if (l >= A.nd) return;
    T* base = sm + A.off[l][arr];
    if (lo > 0) up = cl.map_shared_rank(base + (size_t)(A.rows[l] + 1) * A.n2[l], (unsigned)(rank - 1));
    if (lo + cnt < A.n1[l]) dn = cl.map_shared_rank(base, (unsigned)(rank + 1));
}

// One colour of a red-black sweep on the band (the arithmetic of k_rb_face5; with zero, the
// first colour of a sweep from x = 0, that of k_rb_zero: x = b * idiag, no neighbour read).
template <class T>
__device__ void cl_sweep(const cooperative_groups::cluster_group& cl, T* sm, int rank, const ClusterArgs<T>& A,
                         int l, int col, bool zero = false) {
    int lo, cnt;
    cl_band(A, l, rank, lo, cnt);
    if (cnt == 0) return;
    const int n1 = A.n1[l], n2 = A.n2[l], half = (n2 + 1) / 2;
    T* x = sm + A.off[l][CL_X] + n2;
    const T* b = sm + A.off[l][CL_B];
    const T* tx = sm + A.off[l][CL_TX];
    const T* ty = sm + A.off[l][CL_TY];
    const T* id = sm + A.off[l][CL_ID];
    T *up, *dn;
    cl_halo(cl, sm, rank, A, l, CL_X, lo, cnt, up, dn);
    for (int k = threadIdx.x; k < cnt * half; k += CL_THREADS) {
        const int li = cl_div(k, A.rhalf[l]), i = lo + li, j = 2 * (k - li * half) + ((i + col) & 1);
        if (j >= n2) continue;
        const int c = li * n2 + j;
        T s = b[c];
        if (!zero) {
            if (i > 0) s += tx[c] * x[c - n2];
            if (i < n1 - 1) s += tx[c + n2] * x[c + n2];
            if (j > 0) s += ty[c + li] * x[c - 1];
            if (j < n2 - 1) s += ty[c + li + 1] * x[c + 1];
        }
        s = s * id[c];
        x[c] = s;
        if (li == 0 && up) up[j] = s;
        if (li == cnt - 1 && dn) dn[j] = s;
    }
}

// First half of the restriction: the residual of every band cell of the colour that the sweep
// before it did not update last, to the CTA that owns its coarse row: P for the child on the even
// fine row, Q for the one on the odd row (each coarse cell has one of each), with the halo rows of
// that CTA's neighbours.  Where no colour is skipped, the black cells' go there and the red ones' to P2, Q2.
template <class T, bool ANY>
__device__ void cl_residual(const cooperative_groups::cluster_group& cl, T* sm, int rank, const ClusterArgs<T>& A,
                            int l) {
    int lo, cnt;
    cl_band(A, l, rank, lo, cnt);
    if (cnt == 0) return;
    const int n1 = A.n1[l], n2 = A.n2[l], half = (n2 + 1) / 2, both = ANY && A.zero_color < 0;
    const int c1 = A.n1[l + 1], c2 = A.n2[l + 1], R = A.rows[l + 1];
    const bool spread = l + 1 < A.nd;
    const T* x = sm + A.off[l][CL_X] + n2;
    const T* b = sm + A.off[l][CL_B];
    const T* tx = sm + A.off[l][CL_TX];
    const T* ty = sm + A.off[l][CL_TY];
    const T* dg = sm + A.off[l][CL_DG];
    for (int t = threadIdx.x; t < cnt * half * (1 + both); t += CL_THREADS) {
        const int second = t >= cnt * half, k = t - second * cnt * half, col = both ? 1 - second : 1 - A.zero_color;
        const int li = cl_div(k, A.rhalf[l]), i = lo + li, j = 2 * (k - li * half) + ((i + col) & 1);
        T r = 0;
        if (j < n2) {
            const int c = li * n2 + j;
            r = b[c];
            if (i > 0) r += tx[c] * x[c - n2];
            if (i < n1 - 1) r += tx[c + n2] * x[c + n2];
            if (j > 0) r += ty[c + li] * x[c - 1];
            if (j < n2 - 1) r += ty[c + li + 1] * x[c + 1];
            r = r - dg[c] * x[c];
        }  // else: the aggregate has no such child (odd n2), its residual counts as zero
        const int I = i >> 1, J = j >> 1, o = spread ? I / R : 0, ro = I - o * R;
        auto put = [&](int arr, T v) {
            T* base = sm + A.off[l + 1][arr] + J;
            T* p = base + (size_t)(ro + 1) * c2;
            (o == rank ? p : cl.map_shared_rank(p, (unsigned)o))[0] = v;
            if (spread && ro == 0 && I > 0) cl.map_shared_rank(base + (size_t)(R + 1) * c2, (unsigned)(o - 1))[0] = v;
            if (spread && ro == R - 1 && I < c1 - 1) cl.map_shared_rank(base, (unsigned)(o + 1))[0] = v;
        };
        put(((i & 1) ? CL_Q : CL_P) + 2 * second, r);
        if (i == n1 - 1 && !(i & 1)) put(CL_Q + 2 * second, T(0));  // odd n1: no child on the odd row
    }
}

// Second half: coarse right-hand side of the rows this CTA owns from its own and the
// neighbouring children (the arithmetic of k_restrict5), and the coarse sweep's first colour from
// x = 0 (red: x = b * idiag), or x = 0 where no sweep precedes the correction.  The dense coarsest level
// (last) takes neither.
template <class T, bool ANY>
__device__ void cl_gather(const cooperative_groups::cluster_group& cl, T* sm, int rank, const ClusterArgs<T>& A,
                          int l, bool last) {
    int lo, cnt;
    cl_band(A, l, rank, lo, cnt);
    if (cnt == 0) return;
    const int n1 = A.n1[l], n2 = A.n2[l];
    const size_t ps = (size_t)(A.rows[l] + 2) * n2;
    T* x = sm + A.off[l][CL_X] + n2;
    T* b = sm + A.off[l][CL_B];
    const T* id = sm + A.off[l][CL_ID];
    const T* P = sm + A.off[l][CL_P] + n2;
    const T* Q = sm + A.off[l][CL_Q] + n2;
    const T *wE = sm + A.off[l][CL_W] + n2, *wW = wE + ps, *wN = wW + ps, *wS = wN + ps;
    // which child lies east, west, north, south: the black ones (zero_color 0) or the red ones
    const T *north = A.zero_color == 1 ? Q : P, *south = A.zero_color == 1 ? P : Q;
    // or all four (P: row 0, column 1; Q: 1, 0; P2: 0, 0; Q2: 1, 1)
    const bool both = ANY && A.zero_color < 0;
    const T *P2 = sm + A.off[l][CL_P2] + n2, *Q2 = sm + A.off[l][CL_Q2] + n2;
    auto east = [&](int k) { return both ? Q[k] + Q2[k] : Q[k]; };
    auto west = [&](int k) { return both ? P2[k] + P[k] : P[k]; };
    auto nort = [&](int k) { return both ? P[k] + Q2[k] : north[k]; };
    auto sout = [&](int k) { return both ? P2[k] + Q[k] : south[k]; };
    T *up, *dn;
    cl_halo(cl, sm, rank, A, l, CL_X, lo, cnt, up, dn);
    for (int k = threadIdx.x; k < cnt * n2; k += CL_THREADS) {
        const int li = cl_div(k, A.rn2[l]), j = k - li * n2, i = lo + li;
        const T e = east(k), w = west(k);
        T v = e + w;
        if (!ANY || !A.plain) {
            v = restrict_sum<T>(e, w, nort(k), sout(k), wE[k], wW[k], wN[k], wS[k]);
            if (i > 0) v = fma(wE[k - n2], east(k - n2), v);
            if (i < n1 - 1) v = fma(wW[k + n2], west(k + n2), v);
            if (j > 0) v = fma(wN[k - 1], nort(k - 1), v);
            if (j < n2 - 1) v = fma(wS[k + 1], sout(k + 1), v);
        }
        b[k] = v;
        const bool sweep = !ANY || A.npre > 0;
        if (last || (sweep && ((i + j) & 1))) continue;
        v = sweep ? v * id[k] : T(0);
        x[k] = v;
        if (li == 0 && up) up[j] = v;
        if (li == cnt - 1 && dn) dn[j] = v;
    }
}

// Prolongation of the coarse iterate to the band's cells of the colour that the post-smoothing
// does not overwrite first, or to all of them (colour -1): the arithmetic of k_prolong.
template <class T, bool ANY>
__device__ void cl_prolong5(const cooperative_groups::cluster_group& cl, T* sm, int rank, const ClusterArgs<T>& A,
                            int l, int col) {
    int lo, cnt;
    cl_band(A, l, rank, lo, cnt);
    if (cnt == 0) return;
    const int n2 = A.n2[l], c1 = A.n1[l + 1], c2 = A.n2[l + 1], R = A.rows[l + 1];
    const int per = col < 0 ? n2 : (n2 + 1) / 2;
    const float rper = col < 0 ? A.rn2[l] : A.rhalf[l];
    T* x = sm + A.off[l][CL_X] + n2;
    T* xc = sm + A.off[l + 1][CL_X] + c2;
    T* wc = sm + A.off[l + 1][CL_W] + c2;
    const size_t ps = (size_t)(R + 2) * c2;
    // coarse rows of the band: this CTA's own and its halos' when the bands line up
    const bool local = l >= A.nd || (l + 1 < A.nd && A.rows[l] == 2 * R);
    T *up, *dn;
    cl_halo(cl, sm, rank, A, l, CL_X, lo, cnt, up, dn);
    for (int k = threadIdx.x; k < cnt * per; k += CL_THREADS) {
        const int li = cl_div(k, rper), i = lo + li, j = col < 0 ? k - li * per : 2 * (k - li * per) + ((i + col) & 1);
        if (j >= n2) continue;
        const int I = i >> 1, J = j >> 1;
        const int I2 = (i & 1) ? min(I + 1, c1 - 1) : max(I - 1, 0), J2 = (j & 1) ? min(J + 1, c2 - 1) : max(J - 1, 0);
        const int ex = (i & 1) ? 0 : 1, ey = (j & 1) ? 2 : 3;
        const T *r1, *r2, *w1;
        if (local) {
            const int b0 = (l + 1 < A.nd ? rank : 0) * R;
            r1 = xc + (I - b0) * c2;
            r2 = xc + (I2 - b0) * c2;
            w1 = wc + (I - b0) * c2;
        } else {
            const int o1 = l + 1 < A.nd ? I / R : 0, o2 = l + 1 < A.nd ? I2 / R : 0;
            T* a = xc + (I - o1 * R) * c2;
            T* b = xc + (I2 - o2 * R) * c2;
            T* c = wc + (I - o1 * R) * c2;
            r1 = o1 == rank ? a : cl.map_shared_rank(a, (unsigned)o1);
            r2 = o2 == rank ? b : cl.map_shared_rank(b, (unsigned)o2);
            w1 = o1 == rank ? c : cl.map_shared_rank(c, (unsigned)o1);
        }
        const int c = li * n2 + j;
        T v = x[c];
        if (ANY && A.plain) {
            v += T(0.5625) * r1[J];
            v += T(0.1875) * r2[J];
            v += T(0.1875) * r1[J2];
            v += T(0.0625) * r2[J2];
        } else {
            v = prolong5<T>(v, r1[J], r2[J], r1[J2], w1[ex * ps + J], w1[ey * ps + J]);
        }
        x[c] = v;
        if (li == 0 && up) up[j] = v;
        if (li == cnt - 1 && dn) dn[j] = v;
    }
}

// ---- nine-point levels
// One colour (ci, cj) = (col >> 1, col & 1) of a four-colour Gauss-Seidel sweep of a
// nine-point level on the band: s = b - sum_e a_e x_e over the neighbours in c_off order,
// x = s * idiag (the arithmetic of k_gs4_exp9).  Bands start on even rows, so a band row's
// parity is its global row's.
template <class T>
__device__ void cl_sweep9(const cooperative_groups::cluster_group& cl, T* sm, int rank, const ClusterArgs<T>& A,
                          int l, int col) {
    int lo, cnt;
    cl_band(A, l, rank, lo, cnt);
    if (cnt == 0) return;
    const int n1 = A.n1[l], n2 = A.n2[l], ci = col >> 1, cj = col & 1;
    const size_t ps = (size_t)A.rows[l] * n2;  // plane stride of the staged band
    T* x = sm + A.off[l][CL_X];
    const T* b = sm + A.off[l][CL_B];
    const T* id = sm + A.off[l][CL_ID];
    const T* a9 = sm + A.off[l][CL_TX];
    const T* xup = lo > 0 ? cl_row(cl, sm, rank, A, l, CL_X, lo - 1, n2) : nullptr;
    const T* xdn = lo + cnt < n1 ? cl_row(cl, sm, rank, A, l, CL_X, lo + cnt, n2) : nullptr;
    const int nr = (cnt - ci + 1) / 2, nc = (n2 - cj + 1) / 2;
    for (int k = threadIdx.x; k < nr * nc; k += blockDim.x) {
        const int li = ci + 2 * (k / nc), j = cj + 2 * (k % nc), i = lo + li, c = li * n2 + j;
        T o = 0;
#pragma unroll
        for (int e = 1; e < 9; ++e) {
            const int ii = i + c_off[e][0], jj = j + c_off[e][1];
            if (ii < 0 || ii >= n1 || jj < 0 || jj >= n2) continue;
            const T xv = ii < lo ? xup[jj] : (ii >= lo + cnt ? xdn[jj] : x[(ii - lo) * n2 + jj]);
            o += a9[e * ps + c] * xv;
        }
        x[c] = (b[c] - o) * id[c];
    }
}

// Residual of the band summed over 2x2 aggregates into the coarse right-hand side (owned by
// whichever CTA holds the coarse row); coarse iterate := 0.  The arithmetic of k_restrict9.
template <class T>
__device__ void cl_restrict9(const cooperative_groups::cluster_group& cl, T* sm, int rank, const ClusterArgs<T>& A,
                             int l) {
    int lo, cnt;
    cl_band(A, l, rank, lo, cnt);
    if (cnt == 0) return;
    const int n1 = A.n1[l], n2 = A.n2[l], c2 = A.n2[l + 1];
    const T* x = sm + A.off[l][CL_X];
    const T* b = sm + A.off[l][CL_B];
    const T* a9 = sm + A.off[l][CL_TX];
    const size_t ps = (size_t)A.rows[l] * n2;  // plane stride
    const T* xup = lo > 0 ? cl_row(cl, sm, rank, A, l, CL_X, lo - 1, n2) : nullptr;
    const T* xdn = lo + cnt < n1 ? cl_row(cl, sm, rank, A, l, CL_X, lo + cnt, n2) : nullptr;
    const int I0 = lo >> 1, I1 = (lo + cnt + 1) >> 1;
    for (int k = threadIdx.x; k < (I1 - I0) * c2; k += blockDim.x) {
        const int I = I0 + k / c2, J = k % c2;
        T s = 0;
        for (int a = 0; a < 2; ++a)
            for (int bb = 0; bb < 2; ++bb) {
                const int i = 2 * I + a, j = 2 * J + bb;
                if (i >= n1 || j >= n2) continue;
                const int c = (i - lo) * n2 + j;
                T r = b[c];
                for (int e = 1; e < 9; ++e) {  // as resid9: r = b - sum a_e x_e - a_0 x
                    const int ii = i + c_off[e][0], jj = j + c_off[e][1];
                    if (ii < 0 || ii >= n1 || jj < 0 || jj >= n2) continue;
                    const T xv = ii < lo ? xup[jj] : (ii >= lo + cnt ? xdn[jj] : x[(ii - lo) * n2 + jj]);
                    r -= a9[e * ps + c] * xv;
                }
                s += r - a9[c] * x[c];
            }
        cl_row(cl, sm, rank, A, l + 1, CL_B, I, c2)[J] = s;
        cl_row(cl, sm, rank, A, l + 1, CL_X, I, c2)[J] = T(0);
    }
}

// Bilinear prolongation of the coarse iterate added to the band (the arithmetic of k_prolong9).
template <class T>
__device__ void cl_prolong9(const cooperative_groups::cluster_group& cl, T* sm, int rank, const ClusterArgs<T>& A,
                            int l) {
    int lo, cnt;
    cl_band(A, l, rank, lo, cnt);
    if (cnt == 0) return;
    const int n2 = A.n2[l], c1 = A.n1[l + 1], c2 = A.n2[l + 1];
    T* x = sm + A.off[l][CL_X];
    for (int k = threadIdx.x; k < cnt * n2; k += blockDim.x) {
        const int li = k / n2, j = k - li * n2, i = lo + li;
        const int I = i >> 1, J = j >> 1;
        int I2 = (i & 1) ? I + 1 : I - 1, J2 = (j & 1) ? J + 1 : J - 1;
        if (I2 < 0 || I2 >= c1) I2 = I;
        if (J2 < 0 || J2 >= c2) J2 = J;
        const T* r1 = cl_row(cl, sm, rank, A, l + 1, CL_X, I, c2);
        const T* r2 = cl_row(cl, sm, rank, A, l + 1, CL_X, I2, c2);
        T v = x[k];
        v += T(0.5625) * r1[J];
        v += T(0.1875) * r2[J];
        v += T(0.1875) * r1[J2];
        v += T(0.0625) * r2[J2];
        x[k] = v;
    }
}

// KIND: FACE5 or EXP9 (every level of the cycle).  ANY: any schedule and transfers of five-point levels; without
// it a skipped colour, weighted transfers and a sweep before the correction are taken for granted, as a CG solve has them by
// default (decided at run time they cost that solve 5%: 128^2 step 1020 / 1066 us).
template <class T, int KIND, bool ANY>
__global__ void __launch_bounds__(CL_THREADS) k_cluster_vcycle(const __grid_constant__ ClusterArgs<T> A) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char cl_raw[];
    T* sm = reinterpret_cast<T*>(cl_raw);
    const int rank = (int)cl.block_rank();

    // stage this CTA's bands: operators of every level
    for (int l = 0; l < A.nl; ++l) {
        int lo, cnt;
        cl_band(A, l, rank, lo, cnt);
        if (cnt == 0) continue;
        const int n2 = A.n2[l];
        const size_t n = (size_t)A.n1[l] * n2, at = (size_t)lo * n2, ps = (size_t)A.rows[l] * n2;
        T* tx = sm + A.off[l][CL_TX];
        T* ty = sm + A.off[l][CL_TY];
        T* id = sm + A.off[l][CL_ID];
        T* dg = sm + A.off[l][CL_DG];
        if (KIND == FACE5) {
            if (l > 0 && !(ANY && A.plain)) {
                // the gather reads the rows above and below too
                T* w = sm + A.off[l][CL_W];
                const int first = lo > 0 ? 0 : n2, last = (lo + cnt < A.n1[l] ? cnt + 2 : cnt + 1) * n2;
                for (int e = 0; e < 4; ++e)
                    for (int k = first + threadIdx.x; k < last; k += CL_THREADS)
                        stage_async(w + e * (ps + 2 * n2) + k, A.w4[l] + e * n + at + k - n2);
            }
            if (l + 1 < A.nl) {  // the dense level needs no operator
                for (int k = threadIdx.x; k < (cnt + 1) * n2; k += CL_THREADS) stage_async(tx + k, A.tx[l] + at + k);
                for (int k = threadIdx.x; k < cnt * (n2 + 1); k += CL_THREADS)
                    stage_async(ty + k, A.ty[l] + (size_t)lo * (n2 + 1) + k);
                for (int k = threadIdx.x; k < cnt * n2; k += CL_THREADS) {
                    stage_async(id + k, A.id[l] + at + k);
                    stage_async(dg + k, A.dg[l] + at + k);
                }
            }
        } else if (l + 1 < A.nl) {  // nine planes and 1/diagonal (the dense level needs neither)
            for (int e = 0; e < 9; ++e)
                for (int k = threadIdx.x; k < cnt * n2; k += CL_THREADS) stage_async(tx + e * ps + k, A.a9[l] + e * n + at + k);
            for (int k = threadIdx.x; k < cnt * n2; k += CL_THREADS) stage_async(id + k, A.id[l] + at + k);
        }
    }
    if (rank == 0) {  // the dense inverse of the coarsest level
        double* dinv = reinterpret_cast<double*>(cl_raw + A.dinv_off);
        for (int k = threadIdx.x; k < A.dn * A.dn; k += CL_THREADS) stage_async(dinv + k, A.dinv + k);
    }
    // The operators were complete before the kernel in front of this one began (it does not write
    // them); its output, level 0's right-hand side and iterate, only counts from here on.
    pdl_enter();
    {
        int lo, cnt;
        cl_band(A, 0, rank, lo, cnt);
        const int n2 = A.n2[0];
        const size_t at = (size_t)lo * n2;
        T* x = sm + A.off[0][CL_X];
        T* b = sm + A.off[0][CL_B];
        for (int k = threadIdx.x; k < cnt * n2; k += CL_THREADS) stage_async(b + k, A.b0 + at + k);
        if (KIND != FACE5) {
            for (int k = threadIdx.x; k < cnt * n2; k += CL_THREADS) stage_async(x + k, A.x0 + at + k);
        } else if (!A.zero0 && cnt > 0) {  // with the neighbours' edge rows
            const int first = lo > 0 ? 0 : 1, last = lo + cnt < A.n1[0] ? cnt + 2 : cnt + 1;
            for (int k = first * n2 + threadIdx.x; k < last * n2; k += CL_THREADS) stage_async(x + k, A.x0 + at + k - n2);
        }
    }
    stage_wait();
    cl.sync();
    const double* dinv = reinterpret_cast<const double*>(cl_raw + A.dinv_off);
    const int L = A.nl - 1;
    if (KIND == FACE5) {
        const int keep = A.npost > 0 ? 1 - A.post_first : -1;  // cells that the prolongation corrects
        // down: the first colour of a level below the first was done with its right-hand side (cl_gather)
        for (int l = 0; l < A.nd; ++l) {
            for (int s = l > 0 ? 1 : 0; s < A.npre; ++s) {
                cl_sweep(cl, sm, rank, A, l, s & 1, A.zero0 && s == 0);
                cl.sync();
            }
            cl_residual<T, ANY>(cl, sm, rank, A, l);
            cl.sync();
            if (l + 1 < A.nd) {
                cl_gather<T, ANY>(cl, sm, rank, A, l + 1, false);
                cl.sync();
            }
        }
        // the small levels and the dense solve on CTA 0
        if (rank == 0) {
            for (int l = A.nd; l < L; ++l) {
                cl_gather<T, ANY>(cl, sm, 0, A, l, false);
                __syncthreads();
                for (int s = 1; s < A.npre; ++s) {
                    cl_sweep(cl, sm, 0, A, l, s & 1);
                    __syncthreads();
                }
                cl_residual<T, ANY>(cl, sm, 0, A, l);
                __syncthreads();
            }
            cl_gather<T, ANY>(cl, sm, 0, A, L, true);
            __syncthreads();
            dense_coarse_apply<T>(A.dn, dinv, sm + A.off[L][CL_B], sm + A.off[L][CL_X] + A.n2[L]);
            for (int l = L - 1; l >= A.nd; --l) {
                cl_prolong5<T, ANY>(cl, sm, 0, A, l, keep);
                __syncthreads();
                for (int s = 0; s < A.npost; ++s) {
                    cl_sweep(cl, sm, 0, A, l, (A.post_first + s) & 1);
                    __syncthreads();
                }
            }
        }
        cl.sync();
        // up: levels spread over the cluster
        for (int l = A.nd - 1; l >= 0; --l) {
            cl_prolong5<T, ANY>(cl, sm, rank, A, l, keep);
            cl.sync();
            for (int s = 0; s < A.npost; ++s) {
                cl_sweep(cl, sm, rank, A, l, (A.post_first + s) & 1);
                cl.sync();
            }
        }
    } else {
        for (int l = 0; l < A.nd; ++l) {
            for (int s = 0; s < A.npre; ++s) {
                cl_sweep9(cl, sm, rank, A, l, s & 3);
                cl.sync();
            }
            cl_restrict9(cl, sm, rank, A, l);
            cl.sync();
        }
        if (rank == 0) {
            for (int l = A.nd; l < L; ++l) {
                for (int s = 0; s < A.npre; ++s) {
                    cl_sweep9(cl, sm, 0, A, l, s & 3);
                    __syncthreads();
                }
                cl_restrict9(cl, sm, 0, A, l);
                __syncthreads();
            }
            dense_coarse_apply<T>(A.dn, dinv, sm + A.off[L][CL_B], sm + A.off[L][CL_X]);
            for (int l = L - 1; l >= A.nd; --l) {
                cl_prolong9(cl, sm, 0, A, l);
                __syncthreads();
                for (int s = 0; s < A.npost; ++s) {
                    cl_sweep9(cl, sm, 0, A, l, 3 - (s & 3));
                    __syncthreads();
                }
            }
        }
        cl.sync();
        for (int l = A.nd - 1; l >= 0; --l) {
            cl_prolong9(cl, sm, rank, A, l);
            cl.sync();
            for (int s = 0; s < A.npost; ++s) {
                cl_sweep9(cl, sm, rank, A, l, 3 - (s & 3));
                cl.sync();
            }
        }
    }
    // level-0 band back to global (local shared memory only: no CTA reads a peer after the
    // last barrier)
    int lo, cnt;
    cl_band(A, 0, rank, lo, cnt);
    const T* x = sm + A.off[0][CL_X] + (KIND == FACE5 ? A.n2[0] : 0);
    for (int k = threadIdx.x; k < cnt * A.n2[0]; k += CL_THREADS) A.x0[(size_t)lo * A.n2[0] + k] = x[k];
}
