// shk_resident.cuh -- what the resident solves (shk_resident.cu, shk_mg_resident.cu) share: blocks that
// own strips of whole rows, tagged words exchanged through L2, sums over every block, the operator on a
// thread's two columns, and the CG scalars.
#pragma once

#include <cuda_runtime.h>
#include <float.h>

#include "shk_device.cuh"

namespace shk {

constexpr int kResThreads = 512, kResWarps = kResThreads / 32;

// The strips' geometry and the exchange buffers.
struct ResComm {
    int nx, ny, txp, ty;     // threads per row group (a multiple of 32), row groups per block
    int groups;              // blocks that own strips
    uint4 *red;              // [2][groups][4] tagged partials
    uint4 *halo;             // [2][groups][2][2 * txp] tagged strip-edge rows
    CgDev *cg;
    unsigned int *epoch;     // tags used so far: the solve's word (res_start)
    unsigned int *arrived;   // blocks that have started
    int spin;                // polls before a wait gives up
    int start_spin;          // polls before a block stops waiting for the launch's other blocks to start
    // tests: test_spin polls instead, in block test_block (-1: in every block) from the last sum of iteration
    // test_iter on (0: from the start)
    int test_spin, test_block, test_iter;
    int test_absent;         // tests: this block does not start (-1: none)
};

// A solve's word, `epoch`, moves on by compare-and-swap only, so every block sees the same solve:
//   t             t tags used so far, no solve running (t < kResRunning: res_tags)
//   kResRunning|t every block of the solve that found t has started
//   t' > t        completed, the tags up to t' used
//   kResLost      lost: not every block started in time, or a wait ran out
constexpr unsigned kResRunning = 1u << 31, kResLost = ~0u;

// Starting.  The blocks of a cooperative launch run together, but not from the same moment: another stream's
// kernel may hold some of their SMs for as long as it likes.  So no block polls for another's words before all
// of them have started, and when that takes too long (start_spin) the solve is lost before it began and the
// host turns to the general kernels, whose blocks wait for nobody.  The last block to arrive starts the
// solve.  One thread of each block; false: the block leaves.
__device__ __forceinline__ bool res_start(const ResComm &A, unsigned &tag0) {
    const unsigned t = *(volatile unsigned *)A.epoch;
    tag0 = t;
    if (t == kResLost || A.test_absent == (int)blockIdx.x) return false;
    __threadfence();
    if (atomicAdd(A.arrived, 1u) + 1 == gridDim.x) {
        *(volatile unsigned *)A.arrived = 0;
        __threadfence();
        atomicCAS(A.epoch, t, t | kResRunning);
    }
    for (int i = 0;; i++) {
        const unsigned w = *(volatile unsigned *)A.epoch;
        if (w != t) return w == (t | kResRunning);
        if (i < A.start_spin) continue;
        const unsigned was = atomicCAS(A.epoch, t, kResLost);
        if (was == t) {
            A.cg->fault = kFaultNotStarted;
            A.cg->done = 1;
        }
        return was == (t | kResRunning);
    }
}

// Ending.  The outcome is settled by the first block that swaps the word: to the tags that it used when it has
// completed the last sum, or to kResLost when a wait of its own ran out.  Every block ends here (one thread of it)
// and writes its rows of the head only if the solve was not lost; a block whose wait for the last sum ran out when
// another has completed it writes them too, since it has contributed to that sum and its x is final.
// (A sum that completes has every block's partial, so no later wait can be the one that ran out.)
// The one that settles a completed solve (kResSettled) writes its record.
enum { kResDropped = 0, kResKept, kResSettled };
__device__ __forceinline__ int res_end(const ResComm &A, unsigned t, unsigned last, bool ok) {
    const unsigned to = ok ? last : kResLost, was = atomicCAS(A.epoch, t | kResRunning, to);
    if (was != (t | kResRunning)) return was != kResLost ? kResKept : kResDropped;
    if (ok) return kResSettled;
    A.cg->fault = kFaultWait;
    A.cg->done = 1;
    return kResDropped;
}

// A block's waits (in its shared memory): one that runs out makes the whole block leave.
struct ResWait {
    int abort;               // a wait of this block ran out
    int spin;                // polls that a wait has
    int test_at, test_spin;  // tests: before the last sum of this iteration, this many (0: never)
};
__device__ __forceinline__ bool wait_over(volatile ResWait &W, int polls) {
    if (polls < W.spin && !W.abort) return false;
    W.abort = 1;
    return true;
}
// One thread, at the start and before an iteration's last sum.
__device__ __forceinline__ void wait_start(const ResComm &A, ResWait &W) {
    const bool test = A.test_block < 0 || A.test_block == (int)blockIdx.x;
    W.abort = 0;
    W.spin = test && A.test_iter == 0 ? A.test_spin : A.spin;
    W.test_at = test && A.test_iter > 0 ? A.test_iter : 0;
    W.test_spin = A.test_spin;
}
__device__ __forceinline__ void wait_iteration(ResWait &W, int iter) {
    if (iter == W.test_at) W.spin = W.test_spin;
}

// ---- tagged words -------------------------------------------------------------------------------
// Half a value and a flag in each 8 bytes, both pairs in one 16-byte access: the word format of NCCL's
// low-latency (LL) protocol.
__device__ __forceinline__ void ll_store(uint4 *p, double v, unsigned tag) {
    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(__double2loint(v)), "r"(tag),
                 "r"(__double2hiint(v)), "r"(tag)
                 : "memory");
}

__device__ __forceinline__ bool ll_try(const uint4 *p, unsigned tag, double &v) {
    unsigned lo, t0, hi, t1;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(lo), "=r"(t0), "=r"(hi), "=r"(t1)
                 : "l"(p)
                 : "memory");
    v = __hiloint2double((int)hi, (int)lo);
    return t0 == tag && t1 == tag;
}

// The scalars of the iteration, computed by one thread after a sum and published by a barrier: 16 warps
// dividing for themselves keep the Float64 units busy longer than the barrier takes (us per iteration
// every thread / one thread: 128^2 with R = 2 5.6 / 3.9, 512^2 with R = 2 6.9 / 5.5).
struct CgScalars {
    double alpha, beta, gamma, pnorm2, rz, rr;
    long long iter;
    int done, status;
};
struct ResSums {
    double wred[3][kResWarps];   // a block's warp partials
    double wsum[3][kResWarps];   // every block's partials, summed per polling warp
    CgDev cg;
    CgScalars sc;
    ResWait wait;
    unsigned tag0;               // tags used before this solve
    int kept;                    // the solve has started; at the end: its outcome (res_end)
    int left;                    // wait.abort as the last sum left it, the same for every thread
};

// After p'Ap: alpha, or zero curvature (k_cg_A's test).
__device__ __forceinline__ void scalars_alpha(CgScalars &s, double pAp, double eps_curv) {
    const double lim = eps_curv * s.pnorm2;
    if ((pAp <= lim && fabs(pAp) <= lim) || isnan(pAp)) {
        s.done = 1;
        s.status = SHK_BREAKDOWN;
    }
    s.alpha = s.gamma / pAp;
}
// After r'z, r'r: beta (one thread), and the stopping test (another); cg_iter_finish's formulas.
__device__ __forceinline__ void scalars_beta(CgScalars &s, double rz) {
    const double beta = rz / s.gamma;
    s.pnorm2 = rz + beta * beta * s.pnorm2;
    s.gamma = rz;
    s.beta = beta;
}
__device__ __forceinline__ void scalars_stop(CgScalars &s, const CgDev &cg, double rz, double rr) {
    const bool krylov = cg.stop_rule == SHK_STOP_KRYLOV;
    const double root = sqrt(krylov ? rz : rr);
    const bool solved = root <= (krylov ? cg.eps_stop : cg.rtol * cg.bnorm) || (krylov && root + 1.0 <= 1.0);
    s.rz = rz;
    s.rr = rr;
    s.iter += 1;
    if (isnan(rz) || isnan(rr)) {
        s.done = 1;
        s.status = SHK_BREAKDOWN;
    } else if (solved) {
        s.done = 1;
        s.status = SHK_OK;
    } else if (s.iter >= cg.itmax) {
        s.done = 1;
        s.status = SHK_NOT_CONVERGED;
    }
}
// The start (cg_init_finish) and the record of the solve.
__device__ __forceinline__ void scalars_start(CgScalars &s, CgDev &cg, double rz, double rr, double bb) {
    cg_init_finish(&cg, rz, rr, bb);
    s.gamma = s.pnorm2 = s.rz = rz;
    s.rr = rr;
    s.alpha = s.beta = 0.0;
    s.iter = 0;
    s.done = cg.done;
    s.status = cg.status;
}
__device__ __forceinline__ CgDev scalars_record(const CgScalars &s, CgDev g) {
    g.done = 1;
    g.status = s.status;
    if (s.iter > 0) {
        g.iter = s.iter;
        g.rz_last = s.rz;
        g.rr = sqrt(s.rr);
        g.rnorm = g.stop_rule == SHK_STOP_KRYLOV ? sqrt(s.rz) : g.rr;
        g.gamma = s.gamma;
        g.beta = s.beta;
        g.pNorm2 = s.pnorm2;
        g.first = 0;
    }
    return g;
}
template <int R>
struct Strip {
    int tid, lane, warp, tx, gy, c0, row0;
    bool act;                // owns columns
    bool south, north;       // reads (and publishes) a strip-edge row across the block boundary
    const double *op;        // aP, aE, aN: [array][row][column of the pair][kResThreads]
    double *edge;            // [2 buffers][2 sides][R][kResWarps]
    double *rows;            // [2 buffers][4][kResThreads]: first row (2 planes), last row (2 planes)
    double aS0, aS1;         // the couplings below the first row
};

// The values a thread's columns exchange inside the block before the operator is applied: the outer
// columns of each warp and the first and last row of each row group.
template <int R>
__device__ __forceinline__ void publish_block(const Strip<R> &S, const double (&v)[R][2], int buf, int ty) {
    double *eL = S.edge + buf * 2 * R * kResWarps, *eR = eL + R * kResWarps;
    if (S.lane == 0) {
#pragma unroll
        for (int j = 0; j < R; j++) eL[j * kResWarps + S.warp] = v[j][0];
    }
    if (S.lane == 31) {
#pragma unroll
        for (int j = 0; j < R; j++) eR[j * kResWarps + S.warp] = v[j][1];
    }
    if (ty > 1) {
        double *w = S.rows + buf * 4 * kResThreads + S.tid;
        w[0] = v[0][0];
        w[kResThreads] = v[0][1];
        w[2 * kResThreads] = v[R - 1][0];
        w[3 * kResThreads] = v[R - 1][1];
    }
}

// Rows of the neighbouring row groups of the same block (after the barrier that follows
// publish_block); rows across the block boundary are left as they are.
template <int R>
__device__ __forceinline__ void group_rows(const Strip<R> &S, int buf, int txp, int ty, double (&s)[2], double (&n)[2]) {
    const double *w = S.rows + buf * 4 * kResThreads;
    if (S.gy > 0) {
        s[0] = w[2 * kResThreads + S.tid - txp];
        s[1] = w[3 * kResThreads + S.tid - txp];
    }
    if (S.gy < ty - 1) {
        n[0] = w[S.tid + txp];
        n[1] = w[kResThreads + S.tid + txp];
    }
}

// out(j, y0, y1) for every row: y = A v, subtraction order E, W, N, S (stencil_apply).  Couplings
// across the grid's edge are zero and the values beyond it finite, so no term needs a bounds test.
template <int R, typename Out>
__device__ __forceinline__ void apply_op(const Strip<R> &S, const double (&v)[R][2], const double (&vs)[2],
                                         const double (&vn)[2], int buf, Out out) {
    const double *eL = S.edge + buf * 2 * R * kResWarps, *eR = eL + R * kResWarps;
    double s0 = vs[0], s1 = vs[1], a0 = S.aS0, a1 = S.aS1;
#pragma unroll
    for (int j = 0; j < R; j++) {
        const double c0 = v[j][0], c1 = v[j][1];
        double w = __shfl_up_sync(0xffffffffu, c1, 1), e = __shfl_down_sync(0xffffffffu, c0, 1);
        if (S.lane == 0) w = S.warp > 0 ? eR[j * kResWarps + S.warp - 1] : 0.0;
        if (S.lane == 31) e = S.warp < kResWarps - 1 ? eL[j * kResWarps + S.warp + 1] : 0.0;
        constexpr int T = kResThreads;
        const double *oP = S.op + 2 * j * T + S.tid, *oE = oP + 2 * R * T, *oN = oE + 2 * R * T;
        const double E0 = oE[0], E1 = oE[T], N0 = oN[0], N1 = oN[T];
        const double W0 = S.tx > 0 ? oE[T - 1] : 0.0;
        const double n0 = j < R - 1 ? v[j < R - 1 ? j + 1 : j][0] : vn[0];
        const double n1 = j < R - 1 ? v[j < R - 1 ? j + 1 : j][1] : vn[1];
        double y0 = oP[0] * c0;
        y0 -= E0 * c1;
        y0 -= W0 * w;
        y0 -= N0 * n0;
        y0 -= a0 * s0;
        double y1 = oP[T] * c1;
        y1 -= E1 * e;
        y1 -= E0 * c0;
        y1 -= N1 * n1;
        y1 -= a1 * s1;
        out(j, y0, y1);
        s0 = c0;
        s1 = c1;
        a0 = N0;
        a1 = N1;
    }
}

// Strip-edge rows across block boundaries: publish this block's first and last row, read the
// neighbours' (the same threads do both, so a buffer two events old has been read).
template <int R>
__device__ __forceinline__ void send_rows(const ResComm &A, const Strip<R> &S, const double (&v)[R][2], int buf,
                                          unsigned tag) {
    uint4 *mine = A.halo + (((size_t)buf * A.groups + blockIdx.x) * 2) * (2 * A.txp) + S.c0;
    if (S.south) {
        ll_store(mine, v[0][0], tag);
        ll_store(mine + 1, v[0][1], tag);
    }
    if (S.north) {
        ll_store(mine + 2 * A.txp, v[R - 1][0], tag);
        ll_store(mine + 2 * A.txp + 1, v[R - 1][1], tag);
    }
}

template <int R>
__device__ __forceinline__ void recv_rows(const ResComm &A, const Strip<R> &S, int buf, unsigned tag, double (&s)[2],
                                          double (&n)[2], volatile ResWait &W) {
    const size_t per = 2 * (size_t)(2 * A.txp);
    const uint4 *base = A.halo + (size_t)buf * A.groups * per + S.c0;
    const long blk = blockIdx.x;
    const uint4 *ps = base + (blk - 1) * (long)per + 2 * A.txp, *pn = base + (blk + 1) * (long)per;
    bool s0 = !S.south, s1 = s0, n0 = !S.north, n1 = n0;
    for (int i = 0; !(s0 && s1 && n0 && n1); i++) {
        if (!s0) s0 = ll_try(ps, tag, s[0]);
        if (!s1) s1 = ll_try(ps + 1, tag, s[1]);
        if (!n0) n0 = ll_try(pn, tag, n[0]);
        if (!n1) n1 = ll_try(pn + 1, tag, n[1]);
        if (!(s0 && s1 && n0 && n1) && wait_over(W, i)) break;
    }
}

// The total of a block's (or the polling warps') 16 values, the same bits in every lane.
__device__ __forceinline__ double sum16(const double *w, int lane) {
    double t = w[lane & 15];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// Sums v over every block: block partials, one tagged store per value; `meanwhile` (work that needs
// no total); then every warp polls its share of the blocks' partials, at most one per lane, and the
// warps' sums are added in the same order in every block.  One thread runs fin(totals), another
// fin2(totals), and a barrier publishes what they leave.  Returns false when a wait ran out: to the
// whole block, so the flag is taken between two barriers (a warp that has left the last one may
// already be in its next wait and set it).
template <int NV, typename Mid, typename Fin, typename Fin2>
__device__ __forceinline__ bool all_sum(const ResComm &A, ResSums &sh, int lane, int warp, double (&v)[NV], int buf,
                                        unsigned tag, Mid meanwhile, Fin fin, Fin2 fin2) {
#pragma unroll
    for (int k = 0; k < NV; k++) {
        v[k] = warp_reduce<false>(v[k]);
        if (lane == 0) sh.wred[k][warp] = v[k];
    }
    __syncthreads();
    const int G = A.groups;  // (a block beyond them takes part in the totals without adding to them)
    const bool alone = gridDim.x == 1;
    uint4 *slots = A.red + (size_t)buf * G * 4;
    double t[NV];
    if (warp < 2) {
        const int lost = *(volatile int *)&sh.wait.abort;
#pragma unroll
        for (int k = 0; k < NV; k++) t[k] = sum16(sh.wred[k], lane);
        // (a block whose wait ran out adds nothing: a sum that completes is one of whole partials)
        if (warp == 0 && !alone && (int)blockIdx.x < G && !lost) {
#pragma unroll
            for (int k = 0; k < NV; k++)
                if (lane == k) ll_store(slots + blockIdx.x * 4 + k, t[k], tag);
        }
    }
    meanwhile();
    if (!alone) {
        const int per = (G + kResWarps - 1) / kResWarps, i = warp * per + lane;  // per <= 16
        double x[NV];
#pragma unroll
        for (int k = 0; k < NV; k++) x[k] = 0.0;
        if (lane < per && i < G) {
            for (int n = 0;; n++) {
                bool ok = true;
#pragma unroll
                for (int k = 0; k < NV; k++) ok = ll_try(slots + i * 4 + k, tag, x[k]) && ok;
                if (ok || wait_over(sh.wait, n)) break;
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < NV; k++) {
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) x[k] += __shfl_down_sync(0xffffffffu, x[k], o);
            if (lane == 0) sh.wsum[k][warp] = x[k];
        }
        __syncthreads();
        if (warp < 2) {
#pragma unroll
            for (int k = 0; k < NV; k++) t[k] = sum16(sh.wsum[k], lane);
        }
    }
    if (warp == 0 && lane == 0) fin(t);
    if (warp == 2 && lane == 0) sh.left = *(volatile int *)&sh.wait.abort;
    if (warp == 1 && lane == 0) fin2(t);
    __syncthreads();
    return !*(volatile int *)&sh.left;
}

// h = x + x0 on the thread's cells, x(j) its columns of row j.  The cells' coordinates are formed anew from a
// thread index that the compiler takes for another value: kept from the start, they and what depends on them
// hold registers through the iterations (spill loads of the 7-row Jacobi solve 188 B a thread with
// them, 72 without: 11.3 and 11.0 us an iteration at 1024 x 1024).
template <int R, typename X>
__device__ __forceinline__ void add_to_head(const ResComm &A, int nx, int ny, const double *x0, double *h, X x) {
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    const int c0 = 2 * (tid % A.txp), gy = tid / A.txp, row0 = ((int)blockIdx.x * A.ty + gy) * R;
    if (gy >= A.ty || c0 >= nx) return;
#pragma unroll
    for (int j = 0; j < R; j++) {
        if (row0 + j >= ny) continue;
        const double2 v = x(j);
        const size_t c = (size_t)(row0 + j) * nx + c0;
        h[c] = v.x + x0[c];
        if (c0 + 1 < nx) h[c + 1] = v.y + x0[c + 1];
    }
}

} // namespace shk
