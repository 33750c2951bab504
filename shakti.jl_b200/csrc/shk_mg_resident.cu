// shk_mg_resident.cu -- the multigrid-preconditioned Float64 CG solve of a small grid in one persistent
// kernel.
//
// On grids up to 512 cells wide a multigrid iteration is launches and latencies: at 256^2 six kernels of 5
// to 10 us (staging a tile, two sweeps, a grid reduction) for 0.3 us of memory traffic.  As in
// shk_resident.cu, blocks own strips of whole rows for the whole solve and exchange strip-edge rows and
// sums as tagged words; here they own the strips of every level above the bottom ones as well, and one
// further block holds the bottom levels' operator in its registers (shk_mg_bottom.cuh): it receives the
// finest bottom level's right-hand side word by word, runs the bottom of the V-cycle and hands the
// result back.
//
// An iteration, in us, by the general kernels and here: 64 x 64 26 and 13.6, 128 x 128 30.4 and 17.5,
// 201 x 150 44 and 25.4, 256 x 256 35.2 and 25.5, 385 x 301 51 and 40, 512 x 512 47 and 41.  What is left is
// the chain of about twelve exchanges between blocks (1 to 1.3 us each) and the bottom levels (6.5 us).
//
// Level 0: a thread owns two columns of R rows (whole 2 x 2 aggregates, so it restricts its own residual),
// with r, p, A p and the Float32 operator in registers and the Float64 operator in shared memory.  Coarser
// levels live in shared memory.  The iterates of a level pass through shared memory with one row of the
// neighbouring blocks on each side.  Between two exchanges of rows there is one sweep: down a level, the
// first sweep's input (on level 0 formed from the neighbour's residual, which this block tracks by
// receiving A p while it waits for p'Ap) and its output; up, the prolonged iterate and the first
// sweep's output.
//
// Element for element the arithmetic is that of the general kernels (the Float32 roundings of ax_sm and
// sweep_sm in shk_mg.cu, the Float64 ones of k_cg_matvec_t); only the order of the sums differs.
#include <algorithm>

#include "shk_mg_bottom.cuh"
#include "shk_resident.cuh"

namespace shk {

constexpr int kMgResLevels = 4;  // levels above the bottom ones, at most

struct MgResLevel {
    int nx, ny, rows;       // the level and a block's rows of it
    int off;                // levels >= 1: first byte of its arrays in shared memory
    const float *aE, *aN, *dP, *wD;
    const uint8_t *act;
    uint2 *halo;            // [2][groups][2][pitch] tagged rows
    int pitch;
    unsigned by_nx, by_nxc; // reciprocals of nx and (nx + 1) / 2 (see over)
};

struct MgResArgs : ResComm {
    const double *aP, *aE, *aN, *rhs, *x0;
    double *h;
    double2 *vec;           // x (R = 4), in the threads' order
    const uint8_t *fmask;
    CgDev init;
    double eps_curv;
    int nd;                 // levels above the bottom ones
    MgResLevel lv[kMgResLevels];
    BottomPlan bp;
    uint2 *gather, *scatter;  // the finest bottom level's right-hand side and result, tagged
    float wc;
};

// ---- tagged Float32 words ----------------------------------------------------------------------------
__device__ __forceinline__ void ll_store(uint2 *p, float v, unsigned tag) {
    asm volatile("st.volatile.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(__float_as_uint(v)), "r"(tag) : "memory");
}
__device__ __forceinline__ float ll_wait(const uint2 *p, unsigned tag, volatile ResWait &W) {
    unsigned v = 0, t = 0;
    for (int i = 0;; i++) {
        asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(v), "=r"(t) : "l"(p) : "memory");
        if (t == tag || wait_over(W, i)) break;
    }
    return __uint_as_float(v);
}

// Two words, or two pairs of adjacent words (16-byte aligned), polled together; a null pointer is not read.
__device__ __forceinline__ void ll_wait2(const uint2 *pa, const uint2 *pb, unsigned tag, float &a, float &b, volatile ResWait &W) {
    for (int k = 0;; k++) {
        unsigned va = 0, ta = tag, vb = 0, tb = tag;
        if (pa) asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(va), "=r"(ta) : "l"(pa) : "memory");
        if (pb) asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(vb), "=r"(tb) : "l"(pb) : "memory");
        a = __uint_as_float(va);
        b = __uint_as_float(vb);
        if ((ta == tag && tb == tag) || wait_over(W, k)) break;
    }
}
__device__ __forceinline__ void ll_wait2(const uint4 *pa, const uint4 *pb, unsigned tag, float2 &a, float2 &b, volatile ResWait &W) {
    for (int k = 0;; k++) {
        uint4 x = make_uint4(0, tag, 0, tag), y = x;
        if (pa)
            asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w)
                         : "l"(pa)
                         : "memory");
        if (pb)
            asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(y.x), "=r"(y.y), "=r"(y.z), "=r"(y.w)
                         : "l"(pb)
                         : "memory");
        a = make_float2(__uint_as_float(x.x), __uint_as_float(x.z));
        b = make_float2(__uint_as_float(y.x), __uint_as_float(y.z));
        if ((x.y == tag && x.w == tag && y.y == tag && y.w == tag) || wait_over(W, k)) break;
    }
}
__device__ __forceinline__ void ll_store(uint2 *p, float2 v, unsigned tag) {  // p 16-byte aligned
    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(__float_as_uint(v.x)), "r"(tag),
                 "r"(__float_as_uint(v.y)), "r"(tag)
                 : "memory");
}

// n words at p[i[k]], all requested before any is looked at.
__device__ __forceinline__ void ll_wait_all(const uint2 *p, const int (&i)[8], float (&v)[8], int n, unsigned tag, volatile ResWait &W) {
    for (int k = 0;; k++) {
        unsigned t[8];
        bool all = true;
#pragma unroll
        for (int m = 0; m < 8; m++) {
            unsigned x = 0;
            t[m] = tag;
            if (m < n && i[m] >= 0)
                asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(t[m]) : "l"(p + i[m]) : "memory");
            v[m] = __uint_as_float(x);
        }
#pragma unroll
        for (int m = 0; m < 8; m++) all = all && t[m] == tag;
        if (all || wait_over(W, k)) break;
    }
}

// i / d for i < 2^20 and d <= 2^10, from m = 2^32 / d rounded up.
__device__ __forceinline__ int over(int i, unsigned m) { return m ? (int)__umulhi((unsigned)i, m) : i; }
static unsigned reciprocal_of(int d) { return d > 1 ? (unsigned)(((1ull << 32) + d - 1) / d) : 0; }

// A level >= 1 in shared memory: rows of nx cells, n = rows * nx; N with the row below the strip first,
// the iterates with a row on each side.
struct MgSm {
    float *E, *D, *w, *b, *N, *X0, *X1;
    uint8_t *act;
    int nx, ny, rows, n, y0;  // y0: the strip's first row
    unsigned by_nx;
    __device__ __forceinline__ MgSm(unsigned char *sm, const MgResLevel &V) {
        nx = V.nx;
        by_nx = V.by_nx;
        ny = V.ny;
        rows = V.rows;
        n = nx * rows;
        y0 = (int)blockIdx.x * rows;
        E = reinterpret_cast<float *>(sm + V.off);
        D = E + n;
        w = D + n;
        b = w + n;
        N = b + n;
        X0 = N + n + nx;
        X1 = X0 + n + 2 * nx;
        act = reinterpret_cast<uint8_t *>(X1 + n + 2 * nx);
    }
    static size_t bytes(int nx, int rows) {
        const size_t n = (size_t)nx * rows;
        return (((7 * n + 5 * (size_t)nx) * sizeof(float) + n) + 15) / 16 * 16;
    }
    // A X at cell i = (x, y) of the strip
    __device__ __forceinline__ float ax(const float *X, int i, int x, int y) const {
        const float *c = X + nx + i;
        const float xc = *c;
        float v = __fmul_rn(D[i], xc);
        if (x < nx - 1) v = __fmaf_rn(E[i], __fsub_rn(xc, c[1]), v);
        if (x > 0) v = __fmaf_rn(E[i - 1], __fsub_rn(xc, c[-1]), v);
        if (y0 + y < ny - 1) v = __fmaf_rn(N[nx + i], __fsub_rn(xc, c[nx]), v);
        if (y0 + y > 0) v = __fmaf_rn(N[i], __fsub_rn(xc, c[-nx]), v);
        return v;
    }
};

template <int R>
struct MgResSmem {
    static constexpr size_t f64 = ((size_t)6 * R * kResThreads + 2 * R * kResWarps + 4 * kResThreads) * sizeof(double);
    static size_t x_bytes(int txp, int rows) { return 2 * (size_t)(rows + 2) * (2 * txp) * sizeof(float); }
};

template <int R>
__global__ void __launch_bounds__(kResThreads, 1) k_mg_resident(const __grid_constant__ MgResArgs A) {
    using L = MgResSmem<R>;
    constexpr int T = kResThreads;
    constexpr bool XG = R > 2;  // x in global memory
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ ResSums sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = A.groups, blk = blockIdx.x;
    int rb = 0;
    volatile ResWait &W = sh.wait;
    if (tid == 0) {
        sh.cg = A.init;
        wait_start(A, sh.wait);
        sh.kept = res_start(A, sh.tag0);
    }
    __syncthreads();
    if (!sh.kept) return;
    const unsigned tag0 = sh.tag0;
    unsigned st = tag0, vt = tag0, ht = tag0;  // tags of sums, V-cycles and row exchanges
    auto nothing = [&]() {};
    CgScalars &sc = sh.sc;
    bool ok = true;

    // ---- the block of the bottom levels: V-cycle bottoms, and the sums only to know when to stop --------
    if (blk == G) {
        BotShared &M = *reinterpret_cast<BotShared *>(smem);
        BotOp O;
        bot_load(A.bp, M, O);
        __syncthreads();
        double v3[3] = {0.0, 0.0, 0.0}, v1[1] = {0.0}, v2[2] = {0.0, 0.0};
        for (bool first = true;; first = false) {  // (one place for the V-cycle: its registers stay registers)
            vt++;
            bot_rhs(A.bp, M, O, [&](const int (&i)[8], float (&v)[8], int n) {
                ll_wait_all(A.gather, i, v, n, vt, W);
            });
            __syncthreads();
            if (W.abort) {  // a result from part of a right-hand side is not handed on
                ok = false;
                break;
            }
            bot_run<2>(A.bp, M, O, A.wc, [&](int i, float v) { ll_store(A.scatter + i, v, vt); });
            __syncthreads();
            rb ^= 1;
            if (first)
                ok = all_sum<3>(
                    A, sh, lane, warp, v3, rb, ++st, nothing,
                    [&](double (&t)[3]) { scalars_start(sc, sh.cg, t[0], t[1], t[2]); }, [](double (&)[3]) {});
            else
                ok = all_sum<2>(
                    A, sh, lane, warp, v2, rb, ++st, nothing, [&](double (&t)[2]) { scalars_beta(sc, t[0]); },
                    [&](double (&t)[2]) { scalars_stop(sc, sh.cg, t[0], t[1]); });
            if (!ok || sc.done) break;
            rb ^= 1;
            ok = all_sum<1>(
                A, sh, lane, warp, v1, rb, ++st, nothing,
                [&](double (&t)[1]) {
                    scalars_alpha(sc, t[0], A.eps_curv);
                    wait_iteration(sh.wait, (int)sc.iter + 1);
                },
                [](double (&)[1]) {});
            if (!ok || sc.done) break;
        }
        if (!ok && tid == 0) res_end(A, tag0, kResLost, false);
        return;
    }

    // ---- a strip --------------------------------------------------------------------------------------
    double *smd = reinterpret_cast<double *>(smem);
    Strip<R> S;
    S.tid = tid;
    S.lane = lane;
    S.warp = warp;
    S.tx = tid % A.txp;
    S.gy = tid / A.txp;
    S.c0 = 2 * S.tx;
    S.row0 = (blk * A.ty + S.gy) * R;
    S.act = S.gy < A.ty && S.c0 < A.nx;
    S.south = S.act && S.gy == 0 && blk > 0;
    S.north = S.act && S.gy == A.ty - 1 && blk + 1 < G;
    S.op = smd;
    S.edge = smd + 6 * R * T;
    S.rows = S.edge + 2 * R * kResWarps;
    const int nx = A.nx, ny = A.ny, ty = A.ty, pitch = 2 * A.txp, brows = ty * R;
    float *X0 = reinterpret_cast<float *>(smem + L::f64), *X1 = X0 + (size_t)(brows + 2) * pitch;
    auto valid = [&](int j, int e) { return S.act && S.c0 + e < nx && S.row0 + j < ny; };
    auto cell = [&](int j, int e) { return (size_t)(S.row0 + j) * nx + S.c0 + e; };
    // Float32 operator of the thread's cells; the couplings west of and below them; w beside the strip
    float E[R][2], N[R][2], D[R][2], w[R][2], W0[R], S0[2], ws[2], wn[2];
    unsigned act = 0;
    const MgResLevel &V0 = A.lv[0];
#pragma unroll
    for (int j = 0; j < R; j++) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int k = (2 * j + e) * T + tid;
            const bool in = valid(j, e);
            smd[k] = in ? A.aP[cell(j, e)] : 1.0;
            smd[2 * R * T + k] = in ? A.aE[cell(j, e)] : 0.0;
            smd[4 * R * T + k] = in ? A.aN[cell(j, e)] : 0.0;
            E[j][e] = in ? V0.aE[cell(j, e)] : 0.0f;
            N[j][e] = in ? V0.aN[cell(j, e)] : 0.0f;
            D[j][e] = in ? V0.dP[cell(j, e)] : 0.0f;
            w[j][e] = in ? V0.wD[cell(j, e)] : 0.0f;
            if (in && V0.act[cell(j, e)]) act |= 1u << (2 * j + e);
        }
        W0[j] = S.tx > 0 && valid(j, 0) ? V0.aE[cell(j, -1)] : 0.0f;
    }
#pragma unroll
    for (int e = 0; e < 2; e++) {
        S0[e] = S.row0 > 0 && valid(0, e) ? V0.aN[cell(-1, e)] : 0.0f;
        ws[e] = S.south && valid(0, e) ? V0.wD[cell(-1, e)] : 0.0f;
        wn[e] = S.north && valid(R, e) ? V0.wD[cell(R, e)] : 0.0f;
    }
    S.aS0 = S.row0 > 0 && valid(0, 0) ? A.aN[cell(-1, 0)] : 0.0;
    S.aS1 = S.row0 > 0 && valid(0, 1) ? A.aN[cell(-1, 1)] : 0.0;
    // levels >= 1 and the iterates (zero beyond the strip, the level and the grid)
    for (int i = tid; i < 2 * (brows + 2) * pitch; i += T) X0[i] = 0.0f;
    for (int l = 1; l < A.nd; l++) {
        const MgResLevel &V = A.lv[l];
        const MgSm M(smem, V);
        for (int i = tid; i < M.n; i += T) {
            const int y = M.y0 + i / M.nx;
            const size_t c = (size_t)M.y0 * M.nx + i;
            const bool in = y < M.ny;
            M.E[i] = in ? V.aE[c] : 0.0f;
            M.D[i] = in ? V.dP[c] : 0.0f;
            M.w[i] = in ? V.wD[c] : 0.0f;
            M.N[M.nx + i] = in ? V.aN[c] : 0.0f;
            M.act[i] = in ? V.act[c] : 0;
        }
        for (int x = tid; x < M.nx; x += T) M.N[x] = M.y0 > 0 ? V.aN[(size_t)(M.y0 - 1) * M.nx + x] : 0.0f;
        for (int i = tid; i < 2 * (M.n + 2 * M.nx); i += T) M.X0[i] = 0.0f;
    }

    double r[R][2], p[R][2], q[R][2], xr[XG ? 1 : R][2];
    double rs[2] = {0.0, 0.0}, rn[2] = {0.0, 0.0};  // r on the rows below and above the strip
    double ps[2] = {0.0, 0.0}, pn[2] = {0.0, 0.0}, zs[2] = {0.0, 0.0}, zn[2] = {0.0, 0.0};  // p and z there
    double2 *xg = A.vec + (size_t)blk * T + tid;
    int hb = 0;  // Float64 row buffer in turn
    unsigned dt = 0;  // its last tag
    auto send64 = [&](const double (&v)[R][2]) {
        hb ^= 1;
        dt = ++ht;
        send_rows<R>(A, S, v, hb, dt);
    };
    auto recv64 = [&](double (&s)[2], double (&n)[2]) { recv_rows<R>(A, S, hb, dt, s, n, W); };
    auto share = [&](const double (&v)[R][2], double (&s)[2], double (&n)[2]) {
        publish_block<R>(S, v, 0, ty);
        __syncthreads();
        if (ty > 1) group_rows<R>(S, 0, A.txp, ty, s, n);
    };

    // ---- level 0 helpers: X holds an iterate with a row on each side -------------------------------------
    int lb[kMgResLevels] = {};  // row buffers in turn
    auto at = [&](int j) { return (1 + S.gy * R + j) * pitch + S.c0; };
    auto put0 = [&](float *X, const float (&v)[R][2]) {
        if (S.gy >= ty) return;
#pragma unroll
        for (int j = 0; j < R; j++) *reinterpret_cast<float2 *>(X + at(j)) = make_float2(v[j][0], v[j][1]);
    };
    // v to X with the neighbours' rows beside it (ends in a block barrier)
    auto exchange0 = [&](float *X, const float (&v)[R][2]) {
        const unsigned t = ++ht;
        lb[0] ^= 1;
        uint2 *mine = V0.halo + ((size_t)lb[0] * G + blk) * 2 * pitch + S.c0;
        if (S.south) ll_store(mine, make_float2(v[0][0], v[0][1]), t);
        if (S.north) ll_store(mine + pitch, make_float2(v[R - 1][0], v[R - 1][1]), t);
        put0(X, v);
        if (S.south || S.north) {
            const uint2 *base = V0.halo + (size_t)lb[0] * G * 2 * pitch + S.c0;
            float2 a, b;
            ll_wait2(S.south ? reinterpret_cast<const uint4 *>(base + ((size_t)(blk - 1) * 2 + 1) * pitch) : nullptr,
                     S.north ? reinterpret_cast<const uint4 *>(base + (size_t)(blk + 1) * 2 * pitch) : nullptr, t, a, b,
                     W);
            if (S.south) *reinterpret_cast<float2 *>(X + S.c0) = a;
            if (S.north) *reinterpret_cast<float2 *>(X + (size_t)(brows + 1) * pitch + S.c0) = b;
        }
        __syncthreads();
    };
    // out(j, y0, y1) = A v at the thread's cells, v also in X
    auto apply0 = [&](const float *X, const float (&v)[R][2], auto out) {
        if (S.gy >= ty) return;
        float2 s = *reinterpret_cast<const float2 *>(X + at(0) - pitch);
        const float2 top = *reinterpret_cast<const float2 *>(X + at(R - 1) + pitch);
        float a0 = S0[0], a1 = S0[1];
#pragma unroll
        for (int j = 0; j < R; j++) {
            const float c0 = v[j][0], c1 = v[j][1], xw = X[at(j) - 1], xe = X[at(j) + 2];
            const float n0 = j < R - 1 ? v[j < R - 1 ? j + 1 : j][0] : top.x, n1 = j < R - 1 ? v[j < R - 1 ? j + 1 : j][1] : top.y;
            float y0 = __fmul_rn(D[j][0], c0), y1 = __fmul_rn(D[j][1], c1);
            y0 = __fmaf_rn(E[j][0], __fsub_rn(c0, c1), y0);
            y1 = __fmaf_rn(E[j][1], __fsub_rn(c1, xe), y1);
            y0 = __fmaf_rn(W0[j], __fsub_rn(c0, xw), y0);
            y1 = __fmaf_rn(E[j][0], __fsub_rn(c1, c0), y1);
            y0 = __fmaf_rn(N[j][0], __fsub_rn(c0, n0), y0);
            y1 = __fmaf_rn(N[j][1], __fsub_rn(c1, n1), y1);
            y0 = __fmaf_rn(a0, __fsub_rn(c0, s.x), y0);
            y1 = __fmaf_rn(a1, __fsub_rn(c1, s.y), y1);
            out(j, y0, y1);
            s = make_float2(c0, c1);
            a0 = N[j][0];
            a1 = N[j][1];
        }
    };
    // ---- levels >= 1 ---------------------------------------------------------------------------------------
    // The strip-edge rows of X: sent by the cells' owners as they write (edge), received here (ends in a
    // block barrier).
    auto edge = [&](const MgSm &M, int l, unsigned t, int x, int y, float v) {
        uint2 *mine = A.lv[l].halo + ((size_t)lb[l] * G + blk) * 2 * M.nx;
        if (y == 0 && blk > 0) ll_store(mine + x, v, t);
        if (y == M.rows - 1 && blk + 1 < G) ll_store(mine + M.nx + x, v, t);
    };
    auto edges_in = [&](const MgSm &M, int l, unsigned t, float *X) {
        const uint2 *base = A.lv[l].halo + (size_t)lb[l] * G * 2 * M.nx;
        for (int x = tid; x < M.nx; x += T) {
            float a, b;
            ll_wait2(blk > 0 ? base + ((size_t)(blk - 1) * 2 + 1) * M.nx + x : nullptr,
                     blk + 1 < G ? base + (size_t)(blk + 1) * 2 * M.nx + x : nullptr, t, a, b, W);
            if (blk > 0) X[x] = a;
            if (blk + 1 < G) X[(M.rows + 1) * M.nx + x] = b;
        }
        __syncthreads();
    };
    // f(i, x, y) for the strip's cells of a level
    auto cells = [&](const MgSm &M, auto f) {
        for (int i = tid; i < M.n; i += T) {
            const int y = over(i, M.by_nx);
            if (M.y0 + y < M.ny) f(i, i - y * M.nx, y);
        }
    };
    // one sweep XI -> XO with the rows beside the strip (XO's edge rows exchanged unless last)
    auto sweep = [&](const MgSm &M, int l, const float *XI, float *XO, float s, bool last) {
        if (!last) ++ht, lb[l] ^= 1;
        const unsigned t = ht;
        cells(M, [&](int i, int x, int y) {
            const float v = __fmaf_rn(__fmul_rn(M.w[i], s), __fsub_rn(M.b[i], M.ax(XI, i, x, y)), XI[M.nx + i]);
            XO[M.nx + i] = v;
            if (!last) edge(M, l, t, x, y, v);
        });
        if (last) __syncthreads();
        else edges_in(M, l, t, XO);
    };

    // ---- the V-cycle: q = z = M^-1 r, partials r'z, r'r --------------------------------------------------
    auto vcycle = [&](double (&sum)[2]) {
        float x[R][2], b[R][2];
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                b[j][e] = (float)r[j][e];
                x[j][e] = __fmul_rn(w[j][e], b[j][e]);
            }
        // down: two sweeps from zero, the first one's rows beside the strip from the residual there
        put0(X0, x);
        if (S.south)
            *reinterpret_cast<float2 *>(X0 + S.c0) = make_float2(__fmul_rn(ws[0], (float)rs[0]), __fmul_rn(ws[1], (float)rs[1]));
        if (S.north)
            *reinterpret_cast<float2 *>(X0 + (size_t)(brows + 1) * pitch + S.c0) =
                make_float2(__fmul_rn(wn[0], (float)rn[0]), __fmul_rn(wn[1], (float)rn[1]));
        __syncthreads();
        const float s2 = A.bp.s2;
        {
            float x1[R][2];
            apply0(X0, x, [&](int j, float y0, float y1) {
                x1[j][0] = __fmaf_rn(__fmul_rn(w[j][0], s2), __fsub_rn(b[j][0], y0), x[j][0]);
                x1[j][1] = __fmaf_rn(__fmul_rn(w[j][1], s2), __fsub_rn(b[j][1], y1), x[j][1]);
            });
#pragma unroll
            for (int j = 0; j < R; j++) x[j][0] = S.gy < ty ? x1[j][0] : 0.0f, x[j][1] = S.gy < ty ? x1[j][1] : 0.0f;
        }
        exchange0(X1, x);
        vt++;
        // restriction: the thread's aggregates, south row first
        {
            const int nxc = A.nd > 1 ? A.lv[A.nd > 1 ? 1 : 0].nx : A.bp.lv[0].nx;
            float res[R][2];
            apply0(X1, x, [&](int j, float y0, float y1) {
                res[j][0] = act >> (2 * j) & 1 ? __fsub_rn(b[j][0], y0) : 0.0f;
                res[j][1] = act >> (2 * j + 1) & 1 ? __fsub_rn(b[j][1], y1) : 0.0f;
            });
#pragma unroll
            for (int j = 0; j < R; j += 2) {
                if (!valid(j, 0)) continue;
                float v = 0.0f;
                v += res[j][0];
                v += res[j][1];
                v += res[j + 1][0];
                v += res[j + 1][1];
                const int yc = (S.gy * R + j) / 2;  // the coarse row within the strip
                if (A.nd > 1) MgSm(smem, A.lv[1]).b[yc * nxc + S.tx] = v;
                else ll_store(A.gather + (size_t)(blk * (brows / 2) + yc) * nxc + S.tx, v, vt);
            }
        }
        for (int l = 1; l < A.nd; l++) {
            __syncthreads();  // b
            const MgSm M(smem, A.lv[l]);
            const unsigned t = ++ht;
            lb[l] ^= 1;
            cells(M, [&](int i, int xx, int y) {
                const float v = __fmul_rn(M.w[i], M.b[i]);
                M.X0[M.nx + i] = v;
                edge(M, l, t, xx, y, v);
            });
            edges_in(M, l, t, M.X0);
            sweep(M, l, M.X0, M.X1, s2, false);
            const bool more = l + 1 < A.nd;
            const int nxc = (M.nx + 1) / 2, nyc = (M.ny + 1) / 2, rc = M.rows / 2;
            float *bc = more ? MgSm(smem, A.lv[more ? l + 1 : l]).b : nullptr;
            for (int k = tid; k < nxc * rc; k += T) {
                const int yc = over(k, A.lv[l].by_nxc), xc = k - yc * nxc;
                if (blk * rc + yc >= nyc) continue;
                float v = 0.0f;
#pragma unroll
                for (int f = 0; f < 4; f++) {
                    const int xx = 2 * xc + (f & 1), y = 2 * yc + (f >> 1), i = xx + y * M.nx;
                    if (xx < M.nx && M.y0 + y < M.ny && M.act[i]) v += __fsub_rn(M.b[i], M.ax(M.X1, i, xx, y));
                }
                if (more) bc[k] = v;
                else ll_store(A.gather + (size_t)(blk * rc + yc) * nxc + xc, v, vt);
            }
        }
        // up
        for (int l = A.nd - 1; l >= 1; l--) {
            const MgSm M(smem, A.lv[l]);
            const bool more = l + 1 < A.nd;
            const MgSm C(smem, A.lv[more ? l + 1 : l]);
            const int nxc = (M.nx + 1) / 2;
            const unsigned t = ++ht;
            lb[l] ^= 1;
            cells(M, [&](int i, int xx, int y) {
                float v = M.X1[M.nx + i];
                const int k = (xx >> 1) + (y >> 1) * nxc;
                const float c = more ? C.X0[C.nx + k]
                                     : ll_wait(A.scatter + (size_t)(M.y0 >> 1) * nxc + k, vt, W);
                if (M.act[i]) v = __fmaf_rn(A.wc, c, v);
                M.X0[M.nx + i] = v;
                edge(M, l, t, xx, y, v);
            });
            edges_in(M, l, t, M.X0);
            sweep(M, l, M.X0, M.X1, s2, false);
            sweep(M, l, M.X1, M.X0, 1.0f, true);
        }
        {
            const int nxc = A.nd > 1 ? A.lv[A.nd > 1 ? 1 : 0].nx : A.bp.lv[0].nx;
#pragma unroll
            for (int j = 0; j < R; j += 2) {
                if (!valid(j, 0)) continue;
                const int yc = (S.gy * R + j) / 2;
                float c;
                if (A.nd > 1) c = MgSm(smem, A.lv[1]).X0[(1 + yc) * nxc + S.tx];
                else c = ll_wait(A.scatter + (size_t)(blk * (brows / 2) + yc) * nxc + S.tx, vt, W);
#pragma unroll
                for (int f = 0; f < 4; f++)
                    if (act >> (2 * j + f) & 1) x[j + (f >> 1)][f & 1] = __fmaf_rn(A.wc, c, x[j + (f >> 1)][f & 1]);
            }
        }
        exchange0(X0, x);
        {
            float x2[R][2];
            apply0(X0, x, [&](int j, float y0, float y1) {
                x2[j][0] = __fmaf_rn(__fmul_rn(w[j][0], s2), __fsub_rn(b[j][0], y0), x[j][0]);
                x2[j][1] = __fmaf_rn(__fmul_rn(w[j][1], s2), __fsub_rn(b[j][1], y1), x[j][1]);
            });
#pragma unroll
            for (int j = 0; j < R; j++) x[j][0] = S.gy < ty ? x2[j][0] : 0.0f, x[j][1] = S.gy < ty ? x2[j][1] : 0.0f;
        }
        exchange0(X1, x);
#pragma unroll
        for (int j = 0; j < R; j++) q[j][0] = q[j][1] = 0.0;
        apply0(X1, x, [&](int j, float y0, float y1) {
            q[j][0] = (double)__fmaf_rn(w[j][0], __fsub_rn(b[j][0], y0), x[j][0]);
            q[j][1] = (double)__fmaf_rn(w[j][1], __fsub_rn(b[j][1], y1), x[j][1]);
        });
        send64(q);
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                sum[0] += r[j][e] * q[j][e];
                sum[1] += r[j][e] * r[j][e];
            }
    };
    auto recv_z = [&]() { recv64(zs, zn); };

    // ---- start: r = b - A x0, z, r'z, r'r, b'b (GROUNDED rows) --------------------------------------------
    double bb = 0.0;
    {
        double s2[2], n2[2], v = 0.0;
#pragma unroll
        for (int e = 0; e < 2; e++) {
#pragma unroll
            for (int j = 0; j < R; j++) {
                q[j][e] = valid(j, e) ? A.x0[cell(j, e)] : 0.0;
                p[j][e] = 0.0;
            }
            s2[e] = S.row0 > 0 && valid(-1, e) ? A.x0[cell(-1, e)] : 0.0;
            n2[e] = valid(R, e) ? A.x0[cell(R, e)] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (XG) xg[(size_t)j * G * T] = make_double2(0.0, 0.0);
            else xr[XG ? 0 : j][0] = xr[XG ? 0 : j][1] = 0.0;
        }
        share(q, s2, n2);
        apply_op<R>(S, q, s2, n2, 0, [&](int j, double y0, double y1) {
            const double b0 = valid(j, 0) ? A.rhs[cell(j, 0)] : 0.0, b1 = valid(j, 1) ? A.rhs[cell(j, 1)] : 0.0;
            r[j][0] = b0 + (-1.0) * y0;
            r[j][1] = b1 + (-1.0) * y1;
            if (valid(j, 0) && A.fmask[cell(j, 0)] == M_GROUNDED) v += b0 * b0;
            if (valid(j, 1) && A.fmask[cell(j, 1)] == M_GROUNDED) v += b1 * b1;
        });
        send64(r);
        recv64(rs, rn);
        bb = v;
    }

    // ---- iterations: z = M^-1 r, sums, p, A p, x, r (one place for the V-cycle) ---------------------------
    double alpha = 0.0;
    for (bool first = true;; first = false) {
        double sum[2] = {0.0, 0.0};
        vcycle(sum);
        rb ^= 1;
        if (first) {
            double v[3] = {sum[0], sum[1], bb};
            ok = all_sum<3>(
                A, sh, lane, warp, v, rb, ++st, recv_z,
                [&](double (&t)[3]) { scalars_start(sc, sh.cg, t[0], t[1], t[2]); }, [](double (&)[3]) {});
        } else {
            ok = all_sum<2>(
                A, sh, lane, warp, sum, rb, ++st,
                [&]() {
                    recv_z();
#pragma unroll
                    for (int j = 0; j < R; j++) {
                        if (XG) {
                            const double2 xj = xg[(size_t)j * G * T];
                            xg[(size_t)j * G * T] = make_double2(xj.x + alpha * p[j][0], xj.y + alpha * p[j][1]);
                        } else {
                            xr[XG ? 0 : j][0] = xr[XG ? 0 : j][0] + alpha * p[j][0];
                            xr[XG ? 0 : j][1] = xr[XG ? 0 : j][1] + alpha * p[j][1];
                        }
                    }
                },
                [&](double (&t)[2]) { scalars_beta(sc, t[0]); },
                [&](double (&t)[2]) { scalars_stop(sc, sh.cg, t[0], t[1]); });
        }
        if (!ok || sc.done) break;
        const double beta = sc.beta;
#pragma unroll
        for (int e = 0; e < 2; e++) {
#pragma unroll
            for (int j = 0; j < R; j++) p[j][e] = q[j][e] + beta * p[j][e];
            ps[e] = zs[e] + beta * ps[e];
            pn[e] = zn[e] + beta * pn[e];
        }
        double s2[2] = {ps[0], ps[1]}, n2[2] = {pn[0], pn[1]}, v[1] = {0.0}, as[2] = {0.0, 0.0}, an[2] = {0.0, 0.0};
        share(p, s2, n2);
        apply_op<R>(S, p, s2, n2, 0, [&](int j, double y0, double y1) {
            q[j][0] = y0;
            q[j][1] = y1;
            v[0] += p[j][0] * y0;
            v[0] += p[j][1] * y1;
        });
        send64(q);
        rb ^= 1;
        ok = all_sum<1>(
            A, sh, lane, warp, v, rb, ++st, [&]() { recv64(as, an); },
            [&](double (&t)[1]) {
                scalars_alpha(sc, t[0], A.eps_curv);
                wait_iteration(sh.wait, (int)sc.iter + 1);
            },
            [](double (&)[1]) {});
        if (!ok || sc.done) break;
        alpha = sc.alpha;
#pragma unroll
        for (int e = 0; e < 2; e++) {
#pragma unroll
            for (int j = 0; j < R; j++) r[j][e] = r[j][e] + (-alpha) * q[j][e];
            rs[e] = rs[e] + (-alpha) * as[e];
            rn[e] = rn[e] + (-alpha) * an[e];
        }
    }

    // ---- h = x + x0 (the row exchanges are the most frequent events: their tag is the last) ----------------
    if (tid == 0) sh.kept = res_end(A, tag0, ht, ok);
    __syncthreads();
    if (sh.kept == kResDropped) return;
    add_to_head<R>(A, nx, ny, A.x0, A.h, [&](int j) {
        return XG ? xg[(size_t)j * G * T] : make_double2(xr[XG ? 0 : j][0], xr[XG ? 0 : j][1]);
    });
    if (tid == 0 && sh.kept == kResSettled) *A.cg = scalars_record(sc, sh.cg);
}

// ---------------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------------
static size_t mg_res_smem(const Ctx *c, int R, int txp, int ty, int nd, MgResLevel *lv) {
    const size_t f64 = R == 2 ? MgResSmem<2>::f64 : MgResSmem<4>::f64;
    size_t off = f64 + MgResSmem<2>::x_bytes(txp, ty * R);
    for (int l = 1; l < nd; l++) {
        const int rows = ty * R >> l;
        if (lv) lv[l].off = (int)off;
        off += MgSm::bytes(c->mg[l].nx, rows);
    }
    return std::max(off, sizeof(BotShared));
}

// Geometry (wider grids have more levels above the bottom ones than a strip of the rows that fit a block holds
// whole aggregates of): rows of at most 512 cells, two or four rows per thread, strips whose height is a multiple of
// 2^nd (every level's aggregates inside one block), one block for the bottom levels.  c->mg's sizes are set.
void mg_res_plan(Ctx *c) {
    ResPlan &P = c->mg_res;
    P = ResPlan();
    int strips;
    const int nd = mg_bottom_start(c, &strips);
    if (c->mg_levels < 2 || nd < 1 || nd > kMgResLevels || c->nx > kResThreads) return;
    const int txp = (((c->nx + 1) / 2) + 31) / 32 * 32;
    int ty = 1;
    while (2 * ty * txp <= kResThreads) ty *= 2;
    for (int R : {2, 4}) {
        const int rows = ty * R, blocks = (c->ny + rows - 1) / rows;
        if (rows % (1 << nd) || blocks + 1 > c->num_sms) continue;
        if (mg_res_smem(c, R, txp, ty, nd, nullptr) + 1024 > 227 * 1024) continue;
        P.rows = R;
        P.txp = txp;
        P.ty = ty;
        P.blocks = blocks;
        return;
    }
}

// Bytes of the exchange buffers (tagged words: cleared once) and of the scratch vector.
size_t mg_res_comm_bytes(const Ctx *c) {
    const ResPlan &P = c->mg_res;
    if (!P.blocks) return 0;
    const int nd = mg_bottom_start(c, nullptr);
    size_t b = (size_t)2 * P.blocks * 4 * sizeof(uint4) + (size_t)2 * P.blocks * 2 * (2 * P.txp) * sizeof(uint4);
    for (int l = 0; l < nd; l++)
        b += (size_t)2 * P.blocks * 2 * (l ? (c->mg[l].nx + 1) / 2 * 2 : 2 * P.txp) * sizeof(uint2);
    return b + 2 * (size_t)((c->mg[nd].nx * c->mg[nd].ny + 1) / 2 * 2) * sizeof(uint2);
}
size_t mg_res_vec_bytes(const Ctx *c) {
    return c->mg_res.rows > 2 ? (size_t)c->mg_res.blocks * kResThreads * c->mg_res.rows * sizeof(double2) : 0;
}

template <int R>
static int mg_res_launch(Ctx *c, MgResArgs &a, size_t smem) {
    return res_cooperative(c, (const void *)k_mg_resident<R>, c->mg_res.blocks + 1, &a, smem, "resident multigrid solve launch");
}

bool mg_res_serves(const Ctx *c, const shk_cg_opts *o) {
    return c->mg_res.blocks > 0 && o->precision == SHK_FP64 && o->precond == SHK_PRECOND_MULTIGRID && c->mg_nu == 2;
}

// One solve on the assembled system and its hierarchy (mg_setup).  Asynchronous.
int mg_res_solve(Ctx *c, const CgDev &init, const double *x0) {
    if (int rc = res_tags(c)) return rc;
    const ResPlan &P = c->mg_res;
    MgResArgs a;
    a.nx = c->nx;
    a.ny = c->ny;
    a.txp = P.txp;
    a.ty = P.ty;
    a.groups = P.blocks;
    res_waits(c, a);
    a.nd = mg_bottom_plan(c, &a.bp);
    unsigned char *b = (unsigned char *)c->mg_res_comm;
    auto take = [&](size_t bytes) {
        unsigned char *q = b;
        b += bytes;
        return q;
    };
    a.red = (uint4 *)take((size_t)2 * P.blocks * 4 * sizeof(uint4));
    a.halo = (uint4 *)take((size_t)2 * P.blocks * 2 * (2 * P.txp) * sizeof(uint4));
    for (int l = 0; l < a.nd; l++) {
        const MgLevel &m = c->mg[l];
        MgResLevel &V = a.lv[l];
        V.nx = m.nx;
        V.ny = m.ny;
        V.rows = P.ty * P.rows >> l;
        V.off = 0;
        V.aE = m.aE;
        V.aN = m.aN;
        V.dP = m.dP;
        V.wD = m.wD;
        V.act = m.act;
        V.pitch = l ? m.nx : 2 * P.txp;
        V.by_nx = reciprocal_of(m.nx);
        V.by_nxc = reciprocal_of((m.nx + 1) / 2);
        V.halo = (uint2 *)take((size_t)2 * P.blocks * 2 * (l ? (m.nx + 1) / 2 * 2 : 2 * P.txp) * sizeof(uint2));
    }
    const size_t nb = (size_t)((c->mg[a.nd].nx * c->mg[a.nd].ny + 1) / 2 * 2) * sizeof(uint2);
    a.gather = (uint2 *)take(nb);
    a.scatter = (uint2 *)take(nb);
    a.aP = c->aP;
    a.aE = c->aE;
    a.aN = c->aN;
    a.rhs = c->rhs;
    a.x0 = x0;
    a.h = c->st.h;
    a.vec = c->mg_res_vec;
    a.fmask = c->mask8;
    a.init = init;
    a.eps_curv = DBL_EPSILON;
    a.wc = c->mg_omega_c;
    const size_t smem = mg_res_smem(c, P.rows, P.txp, P.ty, a.nd, a.lv);
    return P.rows == 2 ? mg_res_launch<2>(c, a, smem) : mg_res_launch<4>(c, a, smem);
}

} // namespace shk
