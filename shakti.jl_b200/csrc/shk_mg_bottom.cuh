// shk_mg_bottom.cuh -- the multigrid levels of one block: at most 64 cells a level in one warp, and up to
// three levels above them with 1, 2 and 8 cells per thread (k_mg_bottom's comment in shk_mg.cu
// says why).  Shared by the V-cycle's bottom kernels and the resident multigrid solve.
#pragma once

#include <type_traits>

#include "shk_device.cuh"

namespace shk {

constexpr int kBotThreads = 512;  // k_mg_bottom
constexpr int kBotWarpCells = 64, kBotWarpLevels = 8;

struct BottomLevel {
    int nx, ny, off;  // offset of this level's cells in the shared arrays
};
struct BottomPlan {
    int nlev, total;
    BottomLevel lv[kMgMaxLevels];
    const float *aE[kMgMaxLevels], *aN[kMgMaxLevels], *dP[kMgMaxLevels], *wD[kMgMaxLevels];
    const uint8_t *act[kMgMaxLevels];
    const int *done;
    float s2;  // Lv::s2
    int strips;  // levels above the one-warp ones (k_mg_bottom: 8, 2 and 1 cells per thread, coarsest last)
};

// Iterates lie in shared memory in rows of nx + 2 with a border of zeros, so that a cell reads its
// neighbours without a bounds test (the couplings across the border are zero); the finest level's in rows of
// an even pitch with two such columns on each side.
constexpr int kBotPad1 = 1600, kBotPad2 = 2100, kBotPad8 = 6200, kBotPadWarp = 200;
// Do a level's cells and padded array fit (strip = 0: one warp, 1, 2: columns of 1 and 2 cells, 3: blocks of 8)?
inline bool bot_fits(int nx, int ny, int strip) {
    const long long x = nx, y = ny;
    if (strip == 0) return x * y <= kBotWarpCells && (x + 2) * (y + 2) <= kBotPadWarp;
    if (strip == 1) return x * y <= kBotThreads && (x + 2) * (y + 2) <= kBotPad1;
    if (strip == 2) return x * ((y + 1) / 2) <= kBotThreads && (x + 2) * ((y + 1) / 2 * 2 + 2) <= kBotPad2;
    return (x + 1) / 2 * ((y + 3) / 4) <= kBotThreads && ((x + 1) / 2 * 2 + 4) * ((y + 3) / 4 * 4 + 2) <= kBotPad8;
}

// One level of k_mg_bottom: this thread's column of C cells.
template <int C>
struct BotStrip {
    float E[C], W[C], N[C], D[C], w[C], b[C], x[C], S0;
    unsigned act;
    int nx, ny, ix, iy, c, q;  // the level's size; the column's first cell, in the level and in its array
    int pitch;
    bool on;

    static constexpr int kCells = C;
    __device__ __forceinline__ bool in(int k) const { return on && iy + k < ny; }
    __device__ __forceinline__ int cell(int k) const { return c + k * nx; }
    __device__ __forceinline__ float &rhs(int k) { return b[k]; }
    __device__ __forceinline__ float result(int k) const { return x[k]; }
    __device__ __forceinline__ void load(const BottomPlan &P, int l) {
        nx = P.lv[l].nx;
        ny = P.lv[l].ny;
        pitch = nx + 2;
        const int t = threadIdx.x, j = t / nx;
        ix = t - j * nx;
        iy = j * C;
        on = iy < ny;
        c = ix + iy * nx;
        q = on ? (iy + 1) * pitch + ix + 1 : pitch + 1;
        act = 0;
        const float *aE = P.aE[l], *aN = P.aN[l], *dP = P.dP[l], *wD = P.wD[l];
        const uint8_t *a = P.act[l];
#pragma unroll
        for (int k = 0; k < C; k++) {
            const int g = c + k * nx;
            const bool v = in(k);
            E[k] = v ? aE[g] : 0.0f;
            W[k] = v && ix > 0 ? aE[g - 1] : 0.0f;
            N[k] = v ? aN[g] : 0.0f;
            D[k] = v ? dP[g] : 0.0f;
            w[k] = v ? wD[g] : 0.0f;
            if (v && a[g]) act |= 1u << k;
            x[k] = b[k] = 0.0f;
        }
        S0 = in(0) && iy > 0 ? aN[c - nx] : 0.0f;
    }
    // (cells beyond the level hold zeros and may be written: the arrays have room for whole columns)
    __device__ __forceinline__ void put(float *X) const {
        if (!on) return;
#pragma unroll
        for (int k = 0; k < C; k++) X[q + k * pitch] = x[k];
    }
    // A x at the column's cells; X holds every cell's x.
    __device__ __forceinline__ void apply(const float *X, float (&y)[C]) const {
        const float xs = X[q - pitch], xn = X[q + C * pitch];
#pragma unroll
        for (int k = 0; k < C; k++) {
            const float xe = X[q + k * pitch + 1], xw = X[q + k * pitch - 1], xc = x[k];
            float v = __fmul_rn(D[k], xc);
            v = __fmaf_rn(E[k], __fsub_rn(xc, xe), v);
            v = __fmaf_rn(W[k], __fsub_rn(xc, xw), v);
            v = __fmaf_rn(N[k], __fsub_rn(xc, k < C - 1 ? x[k < C - 1 ? k + 1 : k] : xn), v);
            v = __fmaf_rn(k > 0 ? N[k > 0 ? k - 1 : 0] : S0, __fsub_rn(xc, k > 0 ? x[k > 0 ? k - 1 : 0] : xs), v);
            y[k] = v;
        }
    }
    __device__ __forceinline__ void sweep(const float *X, float s) {
        float y[C];
        apply(X, y);
#pragma unroll
        for (int k = 0; k < C; k++) x[k] = __fmaf_rn(__fmul_rn(w[k], s), __fsub_rn(b[k], y[k]), x[k]);
    }
    // right-hand side from the finer level's residuals R, in rows of pf from column `left`
    __device__ __forceinline__ void gather(const float *R, int pf, int left = 1) {
        if (!on) return;
        const float *f = R + (2 * iy + 1) * pf + 2 * ix + left;
#pragma unroll
        for (int k = 0; k < C; k++, f += 2 * pf) {
            if (!in(k)) continue;
            float v = 0.0f;
            v += f[0];
            v += f[1];
            v += f[pf];
            v += f[pf + 1];
            b[k] = v;
        }
    }
    // descending half: two sweeps from zero, then the residual (0 on inactive cells) in X0
    template <int U, typename Sync>
    __device__ __forceinline__ void down(float *X0, float *X1, float s2, Sync sync) {
#pragma unroll
        for (int k = 0; k < C; k++) x[k] = __fmul_rn(w[k], b[k]);
#pragma unroll U
        for (int half = 0; half < 2; half++) {
            float *X = half ? X1 : X0, y[C];
            put(X);
            sync();
            apply(X, y);
#pragma unroll
            for (int k = 0; k < C; k++) {
                const float d = __fsub_rn(b[k], y[k]);
                if (!half) x[k] = __fmaf_rn(__fmul_rn(w[k], s2), d, x[k]);
                else if (on) X0[q + k * pitch] = act >> k & 1 ? d : 0.0f;
            }
        }
        sync();
    }
    // ascending half: prolongation of the coarse result XC (rows of pc), two sweeps; the result in x
    template <int U, typename Sync>
    __device__ __forceinline__ void up(float *X0, float *X1, const float *XC, int pc, float wc, float s2, Sync sync) {
#pragma unroll
        for (int k = 0; k < C; k++)
            if (act >> k & 1) x[k] = __fmaf_rn(wc, XC[(((iy + k) >> 1) + 1) * pc + (ix >> 1) + 1], x[k]);
#pragma unroll U
        for (int half = 0; half < 2; half++) {
            float *X = half ? X0 : X1;
            put(X);
            sync();
            sweep(X, half ? 1.0f : s2);
        }
    }
};

__device__ __forceinline__ float2 less2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }

// The finest level of k_mg_bottom: this thread's block of two columns and four rows, a row's pair in one
// packed operation.  Iterates lie in rows of `pitch` with two columns of zeros on the left, so that pairs are
// aligned.  A phase at 64 x 64 takes 480 cycles, most of them issue (a column of 8 cells per thread needs twice
// the arithmetic instructions and half as many loads again: an iteration of a solve that holds the bottom
// levels for its whole length, 256 x 256, took 26.4 us with it and takes 25.4 us).
struct BotQuad {
    static constexpr int kCells = 8, kLeft = 2;
    float2 E[4], N[4], D[4], w[4], b[4], x[4], S0;
    float W[4];
    unsigned act;
    int nx, ny, ix, iy, c, q, pitch;
    bool on;

    __device__ __forceinline__ bool in(int k) const { return on && iy + (k >> 1) < ny && ix + (k & 1) < nx; }
    __device__ __forceinline__ int cell(int k) const { return c + (k >> 1) * nx + (k & 1); }
    __device__ __forceinline__ float &rhs(int k) { return k & 1 ? b[k >> 1].y : b[k >> 1].x; }
    __device__ __forceinline__ float result(int k) const { return k & 1 ? x[k >> 1].y : x[k >> 1].x; }
    __device__ __forceinline__ void load(const BottomPlan &P, int l) {
        nx = P.lv[l].nx;
        ny = P.lv[l].ny;
        const int pairs = (nx + 1) / 2, t = threadIdx.x, j = t / pairs;
        pitch = 2 * pairs + 4;
        ix = 2 * (t - j * pairs);
        iy = j * 4;
        on = iy < ny;
        c = ix + iy * nx;
        q = on ? (iy + 1) * pitch + ix + kLeft : pitch + kLeft;
        act = 0;
        const float *aE = P.aE[l], *aN = P.aN[l], *dP = P.dP[l], *wD = P.wD[l];
        const uint8_t *a = P.act[l];
        auto pair = [&](const float *F, int r) {
            return make_float2(in(2 * r) ? F[cell(2 * r)] : 0.0f, in(2 * r + 1) ? F[cell(2 * r + 1)] : 0.0f);
        };
#pragma unroll
        for (int r = 0; r < 4; r++) {
            E[r] = pair(aE, r);
            W[r] = in(2 * r) && ix > 0 ? aE[cell(2 * r) - 1] : 0.0f;
            N[r] = pair(aN, r);
            D[r] = pair(dP, r);
            w[r] = pair(wD, r);
            if (in(2 * r) && a[cell(2 * r)]) act |= 1u << 2 * r;
            if (in(2 * r + 1) && a[cell(2 * r + 1)]) act |= 2u << 2 * r;
            x[r] = b[r] = make_float2(0.0f, 0.0f);
        }
        S0 = make_float2(in(0) && iy > 0 ? aN[c - nx] : 0.0f, in(1) && iy > 0 ? aN[c - nx + 1] : 0.0f);
    }
    __device__ __forceinline__ void put(float *X) const {
        if (!on) return;
#pragma unroll
        for (int r = 0; r < 4; r++) *reinterpret_cast<float2 *>(X + q + r * pitch) = x[r];
    }
    __device__ __forceinline__ void apply(const float *X, float2 (&y)[4]) const {
        const float2 xs = *reinterpret_cast<const float2 *>(X + q - pitch),
                     xn = *reinterpret_cast<const float2 *>(X + q + 4 * pitch);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float xe = X[q + r * pitch + 2], xw = X[q + r * pitch - 1];
            const float2 xc = x[r];
            float2 v = __fmul2_rn(D[r], xc);
            v = __ffma2_rn(E[r], less2(xc, make_float2(xc.y, xe)), v);
            v = __ffma2_rn(make_float2(W[r], E[r].x), less2(xc, make_float2(xw, xc.x)), v);
            v = __ffma2_rn(N[r], less2(xc, r < 3 ? x[r < 3 ? r + 1 : r] : xn), v);
            v = __ffma2_rn(r > 0 ? N[r > 0 ? r - 1 : 0] : S0, less2(xc, r > 0 ? x[r > 0 ? r - 1 : 0] : xs), v);
            y[r] = v;
        }
    }
    __device__ __forceinline__ void sweep(const float *X, float s) {
        float2 y[4];
        apply(X, y);
#pragma unroll
        for (int r = 0; r < 4; r++) x[r] = __ffma2_rn(__fmul2_rn(w[r], make_float2(s, s)), less2(b[r], y[r]), x[r]);
    }
    template <int U, typename Sync>
    __device__ __forceinline__ void down(float *X0, float *X1, float s2, Sync sync) {
#pragma unroll
        for (int r = 0; r < 4; r++) x[r] = __fmul2_rn(w[r], b[r]);
#pragma unroll U
        for (int half = 0; half < 2; half++) {
            float *X = half ? X1 : X0;
            float2 y[4];
            put(X);
            sync();
            apply(X, y);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float2 d = less2(b[r], y[r]);
                if (!half) x[r] = __ffma2_rn(__fmul2_rn(w[r], make_float2(s2, s2)), d, x[r]);
                else if (on)
                    *reinterpret_cast<float2 *>(X0 + q + r * pitch) =
                        make_float2(act >> 2 * r & 1 ? d.x : 0.0f, act >> 2 * r & 2 ? d.y : 0.0f);
            }
        }
        sync();
    }
    template <int U, typename Sync>
    __device__ __forceinline__ void up(float *X0, float *X1, const float *XC, int pc, float wc, float s2, Sync sync) {
#pragma unroll
        for (int r = 0; r < 4; r += 2) {
            const float xc = XC[(((iy + r) >> 1) + 1) * pc + (ix >> 1) + 1];
#pragma unroll
            for (int m = r; m < r + 2; m++) {
                if (act >> 2 * m & 1) x[m].x = __fmaf_rn(wc, xc, x[m].x);
                if (act >> 2 * m & 2) x[m].y = __fmaf_rn(wc, xc, x[m].y);
            }
        }
#pragma unroll U
        for (int half = 0; half < 2; half++) {
            float *X = half ? X0 : X1;
            put(X);
            sync();
            sweep(X, half ? 1.0f : s2);
        }
    }
};

// A one-warp level: per cell the operator with all four couplings (zeros beyond the level), the right-hand
// side, and the cell's place in this level's array, its first child's in the finer level's and its parent's
// in the coarser's.  A level of at most 32 cells lies one cell to a lane and reads its neighbours by
// shuffles (about 110 cycles a phase; with every level in shared memory, bounds tests and the coordinates'
// divisions in every phase the one-warp levels took 20000 cycles a V-cycle, now 2400); its child is then the finer level's lane (bits 5 and 6: the second column, the second row
// exist), its parent the coarser level's lane, and X0 holds its iterate by lanes.
struct BotSmall {
    float E[kBotWarpCells], W[kBotWarpCells], N[kBotWarpCells], S[kBotWarpCells], D[kBotWarpCells], w[kBotWarpCells],
        b[kBotWarpCells];
    float X0[kBotPadWarp], X1[kBotPadWarp];
    uint16_t q[kBotWarpCells], child[kBotWarpCells], parent[kBotWarpCells];
    uint8_t act[kBotWarpCells];
    int nx, n;  // the level's row length and cells
};

struct BotShared {
    float X8[2][kBotPad8], X2[2][kBotPad2], X1[2][kBotPad1];
    BotSmall sm[kBotWarpLevels];
};

// The lane's two cells of a one-warp level of more than 32, in registers for the three phases of a half
// cycle.
struct BotPair {
    float E[2], W[2], N[2], S[2], D[2], w[2], b[2], x[2];
    int q[2], pitch;
    bool on[2], act[2];
    __device__ __forceinline__ void load(const BotSmall &M, int nx, int n, int lane) {
        pitch = nx + 2;
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const int i = lane + 32 * t;
            on[t] = i < n;
            const int k = on[t] ? i : 0;
            E[t] = M.E[k], W[t] = M.W[k], N[t] = M.N[k], S[t] = M.S[k], D[t] = M.D[k], w[t] = M.w[k], b[t] = M.b[k];
            q[t] = M.q[k];
            act[t] = M.act[k] != 0;
        }
    }
    __device__ __forceinline__ void put(float *X) const {
#pragma unroll
        for (int t = 0; t < 2; t++)
            if (on[t]) X[q[t]] = x[t];
        __syncwarp();
    }
    __device__ __forceinline__ float ax(const float *X, int t) const {
        const float *c = X + q[t];
        const float xc = x[t], xe = c[1], xw = c[-1], xn = c[pitch], xs = c[-pitch];
        float y = __fmul_rn(D[t], xc);
        y = __fmaf_rn(E[t], __fsub_rn(xc, xe), y);
        y = __fmaf_rn(W[t], __fsub_rn(xc, xw), y);
        y = __fmaf_rn(N[t], __fsub_rn(xc, xn), y);
        y = __fmaf_rn(S[t], __fsub_rn(xc, xs), y);
        return y;
    }
    __device__ __forceinline__ void sweep(const float *X, float s) {
#pragma unroll
        for (int t = 0; t < 2; t++) x[t] = __fmaf_rn(__fmul_rn(w[t], s), __fsub_rn(b[t], ax(X, t)), x[t]);
    }
};

// b of a one-warp level from the finer level's residuals R, in rows of pf.
__device__ __forceinline__ void bot_gather(BotSmall &M, int n, const float *R, int pf, int lane) {
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const int i = lane + 32 * t;
        if (i >= n) continue;
        const float *f = R + M.child[i];
        float v = 0.0f;
        v += f[0];
        v += f[1];
        v += f[pf];
        v += f[pf + 1];
        M.b[i] = v;
    }
    __syncwarp();
}

// The lane's cell of a level of at most 32.
struct BotLane {
    float E, W, N, S, D, w;
    int nx;
    bool act;
    __device__ __forceinline__ void load(const BotSmall &M, int nx_, int lane) {
        nx = nx_;
        E = M.E[lane], W = M.W[lane], N = M.N[lane], S = M.S[lane], D = M.D[lane], w = M.w[lane];
        act = M.act[lane] != 0;
    }
    __device__ __forceinline__ float ax(float x) const {
        const unsigned all = 0xffffffffu;
        const float xe = __shfl_down_sync(all, x, 1), xw = __shfl_up_sync(all, x, 1);
        const float xn = __shfl_down_sync(all, x, nx), xs = __shfl_up_sync(all, x, nx);
        float y = __fmul_rn(D, x);
        y = __fmaf_rn(E, __fsub_rn(x, xe), y);
        y = __fmaf_rn(W, __fsub_rn(x, xw), y);
        y = __fmaf_rn(N, __fsub_rn(x, xn), y);
        y = __fmaf_rn(S, __fsub_rn(x, xs), y);
        return y;
    }
    __device__ __forceinline__ float sweep(float x, float b, float s) const {
        return __fmaf_rn(__fmul_rn(w, s), __fsub_rn(b, ax(x)), x);
    }
};

// The levels P.strips .. nlev - 1 by one warp; sm[0].b holds the right-hand side, the result ends in
// sm[0].X1.  Only the first level can have more than 32 cells: halving both sides of one of at most 64
// leaves at most 32.
__device__ __forceinline__ void bot_warp(const BottomPlan &P, BotSmall *sm, float wc, int lane) {
    const int n_lv = P.nlev - P.strips;
    const unsigned all = 0xffffffffu;
    const int nx0 = sm[0].nx, n0 = sm[0].n, l0 = n0 > 32 ? 1 : 0;
    BotPair C;
    if (l0) {
        BotSmall &M = sm[0];
        C.load(M, nx0, n0, lane);
#pragma unroll
        for (int t = 0; t < 2; t++) C.x[t] = __fmul_rn(C.w[t], C.b[t]);
        C.put(M.X0);
        C.sweep(M.X0, P.s2);
        C.put(M.X1);
        float r[2];
#pragma unroll
        for (int t = 0; t < 2; t++) r[t] = C.act[t] ? __fsub_rn(C.b[t], C.ax(M.X1, t)) : 0.0f;
#pragma unroll
        for (int t = 0; t < 2; t++)
            if (C.on[t]) M.X0[C.q[t]] = r[t];
        __syncwarp();
        bot_gather(sm[1], sm[1].n, M.X0, nx0 + 2, lane);
    }
    float x = 0.0f, b = lane < sm[l0].n ? sm[l0].b[lane] : 0.0f;
    BotLane A;
#pragma unroll 1
    for (int l = l0; l < n_lv - 1; l++) {
        BotSmall &M = sm[l];
        const int child = sm[l + 1].child[lane], nx = M.nx;
        A.load(M, nx, lane);
        x = __fmul_rn(A.w, b);
        x = A.sweep(x, b, P.s2);
        const float y = A.ax(x), r = A.act ? __fsub_rn(b, y) : 0.0f;
        M.b[lane] = b;
        M.X0[lane] = x;
        const int f = child & 31;
        const float r0 = __shfl_sync(all, r, f), r1 = __shfl_sync(all, r, f + 1), r2 = __shfl_sync(all, r, f + nx),
                    r3 = __shfl_sync(all, r, f + nx + 1);
        const bool e = child & 32, n = child & 64;
        b = 0.0f;
        b += r0;
        b += e ? r1 : 0.0f;
        b += n ? r2 : 0.0f;
        b += e && n ? r3 : 0.0f;
    }
    {  // coarsest level (one cell): exact solve
        const BotSmall &M = sm[n_lv - 1];
        x = M.act[lane] ? b / M.D[lane] : (lane == 0 ? b : 0.0f);
    }
#pragma unroll 1
    for (int l = n_lv - 2; l >= l0; l--) {
        BotSmall &M = sm[l];
        const float xc = __shfl_sync(all, x, M.parent[lane]);
        A.load(M, M.nx, lane);
        b = M.b[lane];
        x = M.X0[lane];
        if (A.act) x = __fmaf_rn(wc, xc, x);
        x = A.sweep(x, b, P.s2);
        x = A.sweep(x, b, 1.0f);
    }
    if (lane < sm[l0].n) sm[l0].X1[sm[l0].q[lane]] = x;
    __syncwarp();
    if (l0) {
        BotSmall &M = sm[0];
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const float xc = sm[1].X1[M.parent[C.on[t] ? lane + 32 * t : 0]];
            if (C.act[t]) C.x[t] = __fmaf_rn(wc, xc, C.x[t]);
        }
        C.put(M.X1);
        C.sweep(M.X1, P.s2);
        C.put(M.X0);
        C.sweep(M.X0, 1.0f);
        C.put(M.X1);
    }
}

// The levels' operators, held for as many solves as follow.
struct BotOp {
    BotQuad A8;
    BotStrip<2> A2;
    BotStrip<1> A1;
};

// A block barrier has to follow.
__device__ __forceinline__ void bot_load(const BottomPlan &P, BotShared &M, BotOp &O) {
    const int tid = threadIdx.x, ns = P.strips;
    if (ns > 2) O.A8.load(P, ns - 3);
    if (ns > 1) O.A2.load(P, ns - 2);
    if (ns > 0) O.A1.load(P, ns - 1);
    auto border = [&](const auto &A, float *X0, float *X1, int rows, int left, int width) {
        for (int i = tid; i < rows + 2; i += kBotThreads) {
            X0[i * A.pitch + left - 1] = X0[i * A.pitch + left + width] = 0.0f;
            X1[i * A.pitch + left - 1] = X1[i * A.pitch + left + width] = 0.0f;
        }
        for (int i = tid; i < width; i += kBotThreads) {
            X0[left + i] = X0[(rows + 1) * A.pitch + left + i] = 0.0f;
            X1[left + i] = X1[(rows + 1) * A.pitch + left + i] = 0.0f;
        }
    };
    if (ns > 2) border(O.A8, M.X8[0], M.X8[1], (O.A8.ny + 3) / 4 * 4, BotQuad::kLeft, (O.A8.nx + 1) / 2 * 2);
    if (ns > 1) border(O.A2, M.X2[0], M.X2[1], (O.A2.ny + 1) / 2 * 2, 1, O.A2.nx);
    if (ns > 0) border(O.A1, M.X1[0], M.X1[1], O.A1.ny, 1, O.A1.nx);
    // one-warp levels: a warp pair per array, every level's load in flight before the first is stored
    const int i = tid & (kBotWarpCells - 1), part = tid / kBotWarpCells;
    float v[kBotWarpLevels];
#pragma unroll
    for (int m = 0; m < kBotWarpLevels; m++) {
        const int l = ns + m;
        v[m] = 0.0f;
        if (l >= P.nlev) continue;
        const int nx = P.lv[l].nx, n = nx * P.lv[l].ny;
        if (i >= n) continue;
        if (part == 0) v[m] = P.aE[l][i];
        if (part == 1) v[m] = P.aN[l][i];
        if (part == 2) v[m] = P.dP[l][i];
        if (part == 3) v[m] = P.wD[l][i];
        if (part == 4) v[m] = P.act[l][i] ? 1.0f : 0.0f;
        if (part == 5 && i % nx > 0) v[m] = P.aE[l][i - 1];
        if (part == 6 && i >= nx) v[m] = P.aN[l][i - nx];
    }
#pragma unroll
    for (int m = 0; m < kBotWarpLevels; m++) {
        const int l = ns + m;
        if (l >= P.nlev) continue;
        BotSmall &S = M.sm[m];
        const int nx = P.lv[l].nx, n = nx * P.lv[l].ny;
        if (tid < kBotPadWarp) S.X0[tid] = S.X1[tid] = 0.0f;
        if (part == 0) S.E[i] = v[m];
        if (part == 1) S.N[i] = v[m];
        if (part == 2) S.D[i] = v[m];
        if (part == 3) S.w[i] = v[m];
        if (part == 4) S.act[i] = v[m] != 0.0f;
        if (part == 5) S.W[i] = v[m];
        if (part == 6) S.S[i] = v[m];
        if (tid == 0) {
            S.nx = nx;
            S.n = n;
        }
        if (part == 7) {
            const int k = i < n ? i : 0, iy = k / nx, ix = k - iy * nx;
            S.q[i] = (uint16_t)((iy + 1) * (nx + 2) + ix + 1);
            int child = 0, parent = 0;
            if (l > 0) {
                const int nf = P.lv[l - 1].nx, mf = P.lv[l - 1].ny;
                if (m > 0 && nf * mf <= 32) child = 2 * iy * nf + 2 * ix + (2 * ix + 1 < nf ? 32 : 0) + (2 * iy + 1 < mf ? 64 : 0);
                else child = (2 * iy + 1) * (nf + 2) + 2 * ix + 1;
            }
            if (l + 1 < P.nlev) {
                const int nc = P.lv[l + 1].nx;
                parent = n <= 32 ? (iy >> 1) * nc + (ix >> 1) : ((iy >> 1) + 1) * (nc + 2) + (ix >> 1) + 1;
            }
            S.child[i] = (uint16_t)child;
            S.parent[i] = (uint16_t)parent;
        }
    }
}

// The finest level's right-hand side: get(cells, values, n) fetches up to 8 of them (cells < 0: none).
template <typename Get>
__device__ __forceinline__ void bot_rhs(const BottomPlan &P, BotShared &M, BotOp &O, Get get) {
    const int ns = P.strips;
    int i[8];
    float v[8];
    auto top = [&](auto &A) {
        constexpr int C = std::remove_reference_t<decltype(A)>::kCells;
#pragma unroll
        for (int k = 0; k < C; k++) i[k] = A.in(k) ? A.cell(k) : -1;
        get(i, v, C);
#pragma unroll
        for (int k = 0; k < C; k++) A.rhs(k) = A.in(k) ? v[k] : 0.0f;
    };
    if (ns == 3) top(O.A8);
    if (ns == 2) top(O.A2);
    if (ns == 1) top(O.A1);
    if (ns == 0) {
        i[0] = (int)threadIdx.x < P.lv[0].nx * P.lv[0].ny ? (int)threadIdx.x : -1;
        get(i, v, 1);
        if (i[0] >= 0) M.sm[0].b[i[0]] = v[0];
    }
}

// One V-cycle (nu = 2) from the right-hand side bot_rhs left and a block barrier after it;
// put(cell, value) for the finest level's cells.  U: sweeps of a half cycle unrolled -- 2 where solves follow
// one another (256 x 256 resident: 25.5 us an iteration, 26.8 with 1), 1 where one solve is a launch and every
// instruction is fetched for the first time (1024 x 1024: a step 1.5 % shorter than with 2).
template <int U, typename Put>
__device__ __forceinline__ void bot_run(const BottomPlan &P, BotShared &M, BotOp &O, float wc, Put put) {
    const int tid = threadIdx.x, ns = P.strips, first = ns;
    BotQuad &A8 = O.A8;
    BotStrip<2> &A2 = O.A2;
    BotStrip<1> &A1 = O.A1;
    auto result = [&](auto &A) {
#pragma unroll
        for (int k = 0; k < std::remove_reference_t<decltype(A)>::kCells; k++)
            if (A.in(k)) put(A.cell(k), A.result(k));
    };
    auto block = [&]() { __syncthreads(); };
    // the one-cell level: the warps that hold cells
    const int n1 = ns > 0 ? A1.nx * A1.ny : 0, t1 = (n1 + 31) / 32 * 32;
    auto some = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(t1) : "memory"); };
    if (ns > 2) {
        A8.down<U>(M.X8[0], M.X8[1], P.s2, block);
        A2.gather(M.X8[0], A8.pitch, BotQuad::kLeft);
    }
    if (ns > 1) {
        A2.down<U>(M.X2[0], M.X2[1], P.s2, block);
        A1.gather(M.X2[0], A2.pitch);
    }
    if (ns > 0 && tid < t1) A1.down<U>(M.X1[0], M.X1[1], P.s2, some);
    if (tid < 32) {
        if (ns > 0) bot_gather(M.sm[0], M.sm[0].n, M.X1[0], A1.pitch, tid);
        bot_warp(P, M.sm, wc, tid);
        if (ns == 0)
            for (int i = tid; i < P.lv[0].nx * P.lv[0].ny; i += 32) put(i, M.sm[0].X1[M.sm[0].q[i]]);
    }
    if (ns == 0) return;
    if (tid < t1) {
        some();
        A1.up<U>(M.X1[0], M.X1[1], M.sm[0].X1, P.lv[first].nx + 2, wc, P.s2, some);
    }
    if (ns == 1) {
        result(A1);
        return;
    }
    if (tid < t1) A1.put(M.X1[1]);
    __syncthreads();
    A2.up<U>(M.X2[0], M.X2[1], M.X1[1], A1.pitch, wc, P.s2, block);
    if (ns == 2) {
        result(A2);
        return;
    }
    A2.put(M.X2[1]);
    __syncthreads();
    A8.up<U>(M.X8[0], M.X8[1], M.X2[1], A2.pitch, wc, P.s2, block);
    result(A8);
}

} // namespace shk
