// The half cycles of mglevel.cuh for large FP32 levels, marching down the rows in registers (included by
// pressure.cu inside namespace impec).
//
// In FP32 the arithmetic of a half cycle is small beside its memory traffic (4096^2: 57 us down, 67 us up
// at the copy bandwidth), yet the shared-memory tiles took 169 and 153 us: 750 issued instructions
// per 64 cells, for staging, index arithmetic, bounds and nine shared loads per update.  Here a warp
// owns a strip of 64 columns, two per lane, and walks down its rows two at a time; each colour
// runs one row behind the one before it (a software pipeline over rows), so that every value it needs is in
// this lane's or a neighbouring lane's registers and every plane is read once, by asynchronous copies three
// steps ahead.  With two rows per step the colours' columns are fixed: on even rows the lane's
// even column is red, on odd rows its odd one.
//
// Measured: 89 us down, 84 up at 4096^2, 26 each at 2048^2 (47 and 42 on tiles).  260 instructions per
// 128 cells at half the issue rate of four warps per scheduler (112 registers): the chain of four
// dependent colours within a step is what is left.  Copies by lane in 8- and 4-byte pieces instead of by
// warp in 16-byte ones: 94 and 91 us; loads into registers one step ahead: 95 and 90.
//
// A colour loses one column at either edge of the strip (the shuffle there has no neighbour) and one row
// at either end of the segment: strips advance by 56 columns, and a segment of H rows reads H + 8.
// Absent cells and faces count as zero, which leaves the sums of the guarded form unchanged.
// Per-cell arithmetic and its order are those of mglevel.cuh: the same bits, and the same packed
// black iterate between the halves.
#pragma once

constexpr int MM_WARPS = 8, MM_COLS = 56;  // warps per block (one strip of one segment each), columns a strip advances
constexpr int MM_MINROWS = 16;              // rows of a segment, at least
constexpr size_t MM_MINCELLS = 3 << 18;      // smaller levels take the tiles (pressure.cu: launch_half)

// One row of a lane's two columns (e: even, o: odd); te, to: west faces; n: north faces.
template <class T>
struct MmRow {
    T be, bo, ie, io, ne, no, te, to;
};

// What a step reads, in a ring of shared memory of the warp's own that asynchronous copies fill
// MM_STAGES - 1 steps ahead.
constexpr int MM_STAGES = 4;
struct MmStage {
    float b[2][64], id[2][64], tx[2][64], ty[2][64];  // rows a, a + 1
    float w[4][32];                                   // transfer weights
    float v[4][32];  // down: diagonals of two rows, 64 columns each; up: two rows of packed black cells, coarse iterate
};
constexpr size_t MM_SMEM = sizeof(MmStage) * MM_STAGES * MM_WARPS;

// N bytes (absent: zeros) to dst; src lies within its array either way.
template <int N>
__device__ __forceinline__ void mm_copy(float* dst, const float* src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(N), "r"(on ? N : 0)
                 : "memory");
}
__device__ __forceinline__ void mm_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// This step's copies of the whole warp have landed, and its reads of the step before are done.
__device__ __forceinline__ void mm_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(MM_STAGES - 2) : "memory");
    __syncwarp();
}

// Rows i, i + 1 of columns c0 .. c0 + 63 of planes with rows of `stride` (n1 rows; columns lo <= c < n2 exist):
// f(r, c, k, on) for every piece of P columns at row r of the two; k: offset of a piece that exists.
template <int P, class F>
__device__ __forceinline__ void mm_pieces(int lane, int n1, int n2, int i, int c0, int stride, int lo, F&& f) {
    constexpr int PR = 64 / P;  // pieces per row
#pragma unroll
    for (int q = 0; q < 2 * PR / 32; ++q) {
        const int r = PR == 16 ? lane >> 4 : q * 32 / PR, c = PR == 16 ? (lane & 15) * P : (lane + q * 32) % PR * P;
        const int ii = min(max(i + r, 0), n1 - 1), j = c0 + c, jj = min(max(j, 0), n2 - P);
        f(r, c, (size_t)ii * stride + jj, i + r >= 0 && i + r < n1 && j >= lo && j < n2);
    }
}
// b, 1/diag, north and west faces of rows a, a + 1.
template <int P>
__device__ __forceinline__ void mm_rows(MmStage& S, int lane, int n1, int n2, int a, int c0, const float* tx, const float* ty,
                                        const float* id, const float* b) {
    mm_pieces<P>(lane, n1, n2, a, c0, n2, 0, [&](int r, int c, size_t k, bool on) {
        mm_copy<4 * P>(&S.b[r][c], b + k, on);
        mm_copy<4 * P>(&S.id[r][c], id + k, on);
        mm_copy<4 * P>(&S.tx[r][c], tx + k, on && a + r > 0);
    });
    mm_pieces<1>(lane, n1, n2, a, c0, n2 + 1, 1, [&](int r, int c, size_t k, bool on) { mm_copy<4>(&S.ty[r][c], ty + k, on); });
}
// A row of 32 coarse (or packed) columns from J0 of a plane with rows of n, N of them: pieces of Q columns.
template <int Q>
__device__ __forceinline__ void mm_half(float* dst, const float* p, int l, int I, int N, int J0, int n) {
    const int J = J0 + l * Q;
    mm_copy<4 * Q>(dst + l * Q, p + (size_t)min(max(I, 0), N - 1) * n + min(max(J, 0), n - Q), I >= 0 && I < N && J >= 0 && J < n);
}
__device__ __forceinline__ MmRow<float> mm_row(const MmStage& S, int lane, int r) {
    const auto at = [&](const float* p) { return reinterpret_cast<const float2*>(p)[lane]; };
    const float2 b = at(S.b[r]), d = at(S.id[r]), n = at(S.tx[r]), t = at(S.ty[r]);
    return {b.x, b.y, d.x, d.y, n.x, n.y, t.x, t.y};
}

// b + t x of the north, south, west and east neighbours.
template <class T>
__device__ __forceinline__ T mm_sum(T b, T tn, T xn, T ts, T xs, T tw, T xw, T te, T xe) {
    T s = b;
    s += tn * xn;
    s += ts * xs;
    s += tw * xw;
    s += te * xe;
    return s;
}

template <class T>
__device__ __forceinline__ T mm_left(T v) { return __shfl_up_sync(0xffffffffu, v, 1); }
template <class T>
__device__ __forceinline__ T mm_right(T v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// H: rows of a segment (even).  bc, xc as in k_down5.
template <int P>
__global__ void __launch_bounds__(32 * MM_WARPS, 2) k_down5_march(int n1, int n2, int H, const float* __restrict__ tx,
                                                                  const float* __restrict__ ty, const float* __restrict__ id,
                                                                  const float* __restrict__ dg, const float* __restrict__ b,
                                                                  float* __restrict__ xp, int n1c, int n2c,
                                                                  const float* __restrict__ w4, float* __restrict__ bc,
                                                                  float* __restrict__ xc) {
    pdl_enter();
    using T = float;
    extern __shared__ __align__(16) unsigned char mm_raw[];
    MmStage* ring = reinterpret_cast<MmStage*>(mm_raw) + (threadIdx.x >> 5) * MM_STAGES;
    const int strips = (n2 + MM_COLS - 1) / MM_COLS, unit = blockIdx.x * MM_WARPS + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31, seg = unit / strips, j = (unit - seg * strips) * MM_COLS - 4 + 2 * lane;
    const int J = j / 2, half = (n2 + 1) / 2, r0 = seg * H, r1 = min(r0 + H, n1);
    if (r0 >= n1) return;  // the whole warp
    const bool e = j >= 0 && j < n2, o = j >= 0 && j + 1 < n2, own = e && lane >= 2 && lane < 30;
    const size_t nc = (size_t)n1c * n2c;
    // for step a: its rows, the diagonals of the black cells of rows a - 3, a - 2, the weights of coarse row
    // I = a / 2 - 2 (plane 1: of row I + 1)
    const int cw = j - 2 * lane, J0 = cw / 2;  // the strip's first columns
    auto issue = [&](int a) {
        MmStage& S = ring[(a / 2) % MM_STAGES];
        if (a < r1 + 4) {
            mm_rows<P>(S, lane, n1, n2, a, cw, tx, ty, id, b);
            mm_pieces<P>(lane, n1, n2, a - 3, cw, n2, 0, [&](int r, int c, size_t k, bool on) { mm_copy<4 * P>(&S.v[2 * r][c], dg + k, on); });
            constexpr int Q = P > 1 ? 2 : 1;
            const int I = a / 2 - 2;
#pragma unroll
            for (int q = 0; q < 4; q += Q) {  // Q planes at a time
                const int p = Q == 2 ? q + (lane >> 4) : q;
                mm_half<Q>(S.w[p], w4 + p * nc, Q == 2 ? lane & 15 : lane, p == 1 ? I + 1 : I, n1c, J0, n2c);
            }
        }
        mm_commit();
    };
    int a = max(r0 - 4, 0);
    for (int s = 0; s < MM_STAGES - 1; ++s) issue(a + 2 * s);
    MmRow<T> q0{}, q1{}, s1{};     // rows a - 2, a - 1, a - 3
    MmRow<T> p0, p1;               // rows a, a + 1
    T u0 = 0, u1 = 0;              // east faces of the odd columns of q0, q1
    T x2e = 0, x1o = 0;            // first red: rows a - 2, a - 1
    T y3e = 0, y2o = 0;            // black: rows a - 3, a - 2
    T z4e = 0, z3o = 0;            // second red: rows a - 4, a - 3
    T f5e = 0, f4o = 0;            // black residual: rows a - 5, a - 4
    T wn = 0, w1 = 0;              // weights: plane 0 of coarse row I - 1, plane 1 of I
    for (; a < r1 + 4; a += 2) {
        mm_wait();
        const MmStage& S = ring[(a / 2) % MM_STAGES];
        p0 = mm_row(S, lane, 0);
        p1 = mm_row(S, lane, 1);
        const float4 w = make_float4(S.w[0][lane], S.w[1][lane], S.w[2][lane], S.w[3][lane]);
        const float2 d = make_float2(S.v[0][2 * lane], S.v[2][2 * lane + 1]);
        issue(a + 2 * (MM_STAGES - 1));  // into the stage read in the step before
        const T t0 = mm_right(p0.te), t1 = mm_right(p1.te);
        const T x0e = p0.be * p0.ie, xo = p1.bo * p1.io;  // first red: rows a, a + 1
        // black: rows a - 1, a
        const T y1e = mm_sum(q1.be, q1.ne, x2e, p0.ne, x0e, q1.te, mm_left(x1o), q1.to, x1o) * q1.ie;
        const T y0o = mm_sum(p0.bo, p0.no, x1o, p1.no, xo, p0.to, x0e, t0, mm_right(x0e)) * p0.io;
        // second red: rows a - 2, a - 1
        const T z2e = mm_sum(q0.be, q0.ne, y3e, q1.ne, y1e, q0.te, mm_left(y2o), q0.to, y2o) * q0.ie;
        const T z1o = mm_sum(q1.bo, q1.no, y2o, p0.no, y0o, q1.to, y1e, u1, mm_right(y1e)) * q1.io;
        // residual of the black cells of rows a - 3, a - 2
        const T f3e = mm_sum(s1.be, s1.ne, z4e, q0.ne, z2e, s1.te, mm_left(z3o), s1.to, z3o) - d.x * y3e;
        const T f2o = mm_sum(q0.bo, q0.no, z3o, q1.no, z1o, q0.to, z2e, u0, mm_right(z2e)) - d.y * y2o;
        if (own) {
            if (a - 3 >= r0 && a - 3 < r1) xp[(size_t)(a - 3) * half + J] = y3e;
            if (o && a - 2 >= r0 && a - 2 < r1) xp[(size_t)(a - 2) * half + J] = y2o;
        }
        // coarse row I = a / 2 - 2: its children's rows a - 4, a - 3 and the rows on either side
        const T fl = mm_left(f4o), fr = mm_right(f3e), ww = mm_left(w.z), we = mm_right(w.w);
        const int I = a / 2 - 2;
        if (own && I >= r0 / 2 && I < n1c) {
            T v = restrict_sum<T>(f3e, f4o, f4o, f3e, w.x, w1, w.z, w.w);
            v = fma(wn, f5e, v);
            v = fma(w.y, f2o, v);
            v = fma(ww, fl, v);
            v = fma(we, fr, v);
            const size_t kk = (size_t)I * n2c + J;
            bc[kk] = v;
            if (xc) xc[kk] = T(0);
        }
        wn = w.x; w1 = w.y;
        x2e = x0e; x1o = xo;
        z4e = z2e; z3o = z1o;
        y3e = y1e; y2o = y0o;
        f5e = f3e; f4o = f2o;
        s1 = q1;
        q0 = p0; q1 = p1; u0 = t0; u1 = t1;
    }
}

template <int P>
__global__ void __launch_bounds__(32 * MM_WARPS, 2) k_up5_march(int n1, int n2, int H, const float* __restrict__ tx,
                                                                const float* __restrict__ ty, const float* __restrict__ id,
                                                                const float* __restrict__ b, const float* __restrict__ xp,
                                                                float* __restrict__ x, int n1c, int n2c,
                                                                const float* __restrict__ xc, const float* __restrict__ w4) {
    pdl_enter();
    using T = float;
    extern __shared__ __align__(16) unsigned char mm_raw[];
    MmStage* ring = reinterpret_cast<MmStage*>(mm_raw) + (threadIdx.x >> 5) * MM_STAGES;
    const int strips = (n2 + MM_COLS - 1) / MM_COLS, unit = blockIdx.x * MM_WARPS + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31, seg = unit / strips, j = (unit - seg * strips) * MM_COLS - 4 + 2 * lane;
    const int J = j / 2, half = (n2 + 1) / 2, r0 = seg * H, r1 = min(r0 + H, n1);
    if (r0 >= n1) return;  // the whole warp
    const bool e = j >= 0 && j < n2, o = j >= 0 && j + 1 < n2, own = e && lane >= 2 && lane < 30;
    const size_t nc = (size_t)n1c * n2c;
    // for step a, I = a / 2: its rows, the packed black cells of rows a (odd column) and a + 1 (even column), the
    // weights of coarse row I and the coarse iterate of row I + 1
    const int cw = j - 2 * lane, J0 = cw / 2;  // the strip's first columns
    auto issue = [&](int a) {
        MmStage& S = ring[(a / 2) % MM_STAGES];
        if (a < r1 + 4) {
            mm_rows<P>(S, lane, n1, n2, a, cw, tx, ty, id, b);
            constexpr int Q = P > 1 ? 2 : 1;
            const int I = a / 2, l = Q == 2 ? lane & 15 : lane;
#pragma unroll
            for (int q = 0; q < 4; q += Q) {  // Q planes at a time
                const int p = Q == 2 ? q + (lane >> 4) : q;
                mm_half<Q>(S.w[p], w4 + p * nc, l, I, n1c, J0, n2c);
                if (p < 2) mm_half<Q>(S.v[p], xp, l, a + p, n1, J0, half);
                else if (p == 2) mm_half<Q>(S.v[p], xc, l, I + 1, n1c, J0, n2c);
            }
        }
        mm_commit();
    };
    int a = max(r0 - 4, 0);
    for (int s = 0; s < MM_STAGES - 1; ++s) issue(a + 2 * s);
    auto coarse = [&](int I) { return e && I >= 0 && I < n1c ? xc[(size_t)I * n2c + J] : T(0); };
    T cm = coarse(a / 2 - 1), c0 = coarse(a / 2);  // coarse rows I - 1, I
    MmRow<T> q0{}, q1{}, s1{};                     // rows a - 2, a - 1, a - 3
    MmRow<T> p0, p1;                               // rows a, a + 1
    T u0 = 0, u1 = 0, s1t = 0;                     // east faces of the odd columns of q0, q1, s1
    T v2o = 0, v1e = 0;                            // corrected black: rows a - 2, a - 1
    T x2e = 0, x3o = 0;                            // first red: rows a - 2, a - 3
    T y3e = 0, y4o = 0;                            // black: rows a - 3, a - 4
    for (; a < r1 + 4; a += 2) {
        mm_wait();
        const MmStage& S = ring[(a / 2) % MM_STAGES];
        p0 = mm_row(S, lane, 0);
        p1 = mm_row(S, lane, 1);
        const float4 w = make_float4(S.w[0][lane], S.w[1][lane], S.w[2][lane], S.w[3][lane]);
        const float4 v = make_float4(S.v[0][lane], S.v[1][lane], S.v[2][lane], 0.f);
        issue(a + 2 * (MM_STAGES - 1));  // into the stage read in the step before
        const T t0 = mm_right(p0.te), t1 = mm_right(p1.te);
        const int I = a / 2;
        // corrected black cells of rows a (odd column) and a + 1 (even column)
        const T cr = mm_right(c0), cl = mm_left(c0);
        T v0o = T(0), ve = T(0);
        if (o && a < n1) v0o = prolong5<T>(v.x, c0, I > 0 ? cm : c0, J + 1 < n2c ? cr : c0, w.y, w.z);
        if (e && a + 1 < n1) ve = prolong5<T>(v.y, c0, I + 1 < n1c ? v.z : c0, J > 0 ? cl : c0, w.x, w.w);
        // first red: rows a - 1, a
        const T x1o = mm_sum(q1.bo, q1.no, v2o, p0.no, v0o, q1.to, v1e, u1, mm_right(v1e)) * q1.io;
        const T x0e = mm_sum(p0.be, p0.ne, v1e, p1.ne, ve, p0.te, mm_left(v0o), p0.to, v0o) * p0.ie;
        // black: rows a - 2, a - 1
        const T y2o = mm_sum(q0.bo, q0.no, x3o, q1.no, x1o, q0.to, x2e, u0, mm_right(x2e)) * q0.io;
        const T y1e = mm_sum(q1.be, q1.ne, x2e, p0.ne, x0e, q1.te, mm_left(x1o), q1.to, x1o) * q1.ie;
        // second red: rows a - 3, a - 2
        const T z3o = mm_sum(s1.bo, s1.no, y4o, q0.no, y2o, s1.to, y3e, s1t, mm_right(y3e)) * s1.io;
        const T z2e = mm_sum(q0.be, q0.ne, y3e, q1.ne, y1e, q0.te, mm_left(y2o), q0.to, y2o) * q0.ie;
        if (own) {
            auto put = [&](int i, T xe, T xo) {
                const size_t k = (size_t)i * n2 + j;
                if (P > 1) {
                    *reinterpret_cast<float2*>(x + k) = make_float2(xe, xo);
                } else {
                    x[k] = xe;
                    if (o) x[k + 1] = xo;
                }
            };
            if (a - 3 >= r0 && a - 3 < r1) put(a - 3, y3e, z3o);
            if (a - 2 >= r0 && a - 2 < r1) put(a - 2, z2e, y2o);
        }
        v2o = v0o; v1e = ve;
        x2e = x0e; x3o = x1o;
        y4o = y2o; y3e = y1e;
        cm = c0; c0 = v.z;
        s1 = q1; s1t = u1;
        q0 = p0; q1 = p1; u0 = t0; u1 = t1;
    }
}
