// shk_resident.cu -- a whole preconditioned Float64 CG solve in one persistent kernel, for grids whose
// Krylov state fits on the chip.
//
// A 1024 x 1024 solve touches r, p, A p (or z), x and the operator aP, aE, aN: 56 B per cell, 59 MB,
// which is less than the 148 SMs hold in registers and shared memory (71 MB).  Launched as two (Jacobi)
// or six (Chebyshev) kernels per iteration, such a solve spends its time on launches, on block
// start-up and on moving those arrays through L2: 20 us per iteration at 201 x 150 and 31 us at 1024^2
// with Jacobi, 25 and 84 us at 64^2 and 1024^2 with Chebyshev(4); here it is 4.4 and 11.8, 6.8 and 26 (a step's
// Picard work and Lanczos bounds not counted).  One block per SM (a cooperative launch) owns a strip of whole
// rows for the entire solve; each thread owns two adjacent columns of R rows, with the operator in shared
// memory and p, A p (z) in registers; r and x are there too for R <= 4 (Jacobi) and R <= 2 (Chebyshev).  For
// larger R the vectors that do not fit lie in shared memory (r; ResSmem) or in a scratch array in L2 in the
// threads' own order (x, and at R = 7 of Chebyshev r and p), each read and written once an iteration.  Otherwise
// only sums and strip-edge rows cross L2.
//
// An iteration has the two all-block sums of CG (p'Ap, then r'z and r'r) and, per application of the
// operator, one exchange of strip-edge rows between neighbours.  Every exchanged Float64 travels as two
// 8-byte words, each carrying half of the value and a 32-bit tag that is new for every event: a reader
// polls the words themselves, so no fence, counter or second round trip stands between a producer and
// its reader, and a block learns every other block's partial one L2 hop after it was written.  A
// buffer is rewritten only two events later, when its readers have provably read it (they contributed
// to the event in between).  Each block adds the partials in the same order, so all blocks take the
// same decisions and stop together.  Polls are bounded, and they begin only when every block of the launch
// runs; how a solve starts, and how it ends when a wait runs out, is told in shk_resident.cuh.
//
// Element for element the arithmetic is that of the general kernels in shk_krylov.cu (same formulas,
// same order, unfused); only the order of the sums differs.
#include <cuda_runtime.h>
#include <float.h>

#include <algorithm>
#include <type_traits>

#include "shk_cheb.cuh"
#include "shk_resident.cuh"

namespace shk {

struct ResArgs : ResComm {
    int deg, nsteps;         // Chebyshev degree and Lanczos steps (0: Jacobi)
    const double *aP, *aE, *aN, *rhs, *x0;
    double *h;
    const uint8_t *fmask;
    CgDev init;
    ChebDev *cheb;
    double2 *vec;            // scratch vectors of the largest R, in the threads' order
    double eps_curv;
};

struct ResCheb {
    double gamma;
    double alphas[kMaxChebSteps], betas[kMaxChebSteps], d[kMaxChebSteps], e[kMaxChebSteps];  // Lanczos
    double ca[kMaxChebDegree + 1], cb[kMaxChebDegree + 1];
    double lam_min, lam_max, est_min, est_max;
    int adopted;
};

// Where a vector lives.  Registers hold what the iteration needs at once; the rest goes to shared
// memory while it lasts (the operator takes 24 B per cell of it), then to a scratch array that stays
// in L2, in the threads' own order, touched once per iteration while the block waits for a sum.
enum { V_REG, V_SMEM, V_GLOBAL };

template <int MODE, int R>
struct ResVec {
    double v[MODE == V_REG ? R : 1][2];
    double *s;        // V_SMEM: this thread's first value, planes of kResThreads
    double2 *g;       // V_GLOBAL: this thread's first pair
    size_t stride;    // V_GLOBAL: pairs from one row to the next
    __device__ __forceinline__ double2 get(int j) const {
        if (MODE == V_GLOBAL) return g[j * stride];
        if (MODE == V_SMEM) return make_double2(s[2 * j * kResThreads], s[(2 * j + 1) * kResThreads]);
        return make_double2(v[MODE == V_REG ? j : 0][0], v[MODE == V_REG ? j : 0][1]);
    }
    __device__ __forceinline__ void set(int j, double a, double b) {
        if (MODE == V_GLOBAL) g[j * stride] = make_double2(a, b);
        if (MODE == V_SMEM) s[2 * j * kResThreads] = a, s[(2 * j + 1) * kResThreads] = b;
        if (MODE == V_REG) v[MODE == V_REG ? j : 0][0] = a, v[MODE == V_REG ? j : 0][1] = b;
    }
};

// Rows per thread and the vectors' places.  At R = 7 (Jacobi) p and A p fill the registers, r the shared
// memory beside the operator, and x is left to L2, whose 17 MB per iteration take 2.6 us of the 11.8 at
// 1024^2; the 14 divides a thread take 3.
template <int R, bool CHEB>
struct ResSmem {
    static constexpr int rmode = R <= (CHEB ? 2 : 4) ? V_REG : (R <= 4 || !CHEB ? V_SMEM : V_GLOBAL);
    static constexpr int xmode = R <= (CHEB ? 2 : 4) ? V_REG : V_GLOBAL;
    static constexpr int pmode = CHEB && R > 4 ? V_GLOBAL : V_REG;
    static constexpr int bufs = CHEB ? 2 : 1;
    // rows with a stored reciprocal of aP, a fourth operator array: all that fit
    static constexpr int recip = R <= 4 ? R : (CHEB ? R - 1 : 0);
    static constexpr int op = 6 * R + 2 * recip;   // operator planes
    static constexpr size_t planes = (size_t)(op + 2 * (rmode == V_SMEM) * R) * kResThreads;
    static constexpr size_t edges = (size_t)bufs * 2 * R * kResWarps;
    static constexpr size_t rows = R > 4 ? 0 : (size_t)bufs * 4 * kResThreads;  // R = 7: one row group
    static constexpr size_t bytes = (planes + edges + rows) * sizeof(double);
};

template <int R, bool CHEB>
__global__ void __launch_bounds__(kResThreads, 1) k_cg_resident(const __grid_constant__ ResArgs A) {
    using L = ResSmem<R, CHEB>;
    constexpr int T = kResThreads;
    extern __shared__ __align__(16) double sm[];
    __shared__ ResSums sh;
    __shared__ typename std::conditional<CHEB, ResCheb, int>::type ch_mem;
    ResCheb &ch = reinterpret_cast<ResCheb &>(ch_mem);  // Chebyshev only
    Strip<R> S;
    S.tid = threadIdx.x;
    S.lane = S.tid & 31;
    S.warp = S.tid >> 5;
    S.tx = S.tid % A.txp;
    S.gy = S.tid / A.txp;
    S.c0 = 2 * S.tx;
    S.row0 = ((int)blockIdx.x * A.ty + S.gy) * R;
    S.act = S.gy < A.ty && S.c0 < A.nx;
    S.south = S.act && S.gy == 0 && blockIdx.x > 0;
    S.north = S.act && S.gy == A.ty - 1 && blockIdx.x + 1 < gridDim.x;
    S.op = sm;
    S.edge = sm + L::planes;
    S.rows = S.edge + L::edges;
    ResVec<L::rmode, R> r;
    ResVec<L::xmode, R> x;
    ResVec<L::pmode, R> pm;  // V_REG: unused, p itself is in registers
    r.s = sm + L::op * T + S.tid;
    x.stride = pm.stride = r.stride = (size_t)gridDim.x * T;
    x.g = A.vec + (size_t)blockIdx.x * T + S.tid;
    pm.g = x.g + R * x.stride;
    r.g = pm.g + R * x.stride;
    const int nx = A.nx, ny = A.ny, ty = R > 4 ? 1 : A.ty;
    int hb = 0, rb = 0, sb = 0;  // halo, sum and shared-memory buffers in turn
    if (S.tid == 0) {
        sh.cg = A.init;
        wait_start(A, sh.wait);
        sh.kept = res_start(A, sh.tag0);
        if (CHEB) {
            ch.lam_min = A.cheb->lam_min;
            ch.lam_max = A.cheb->lam_max;
        }
    }
    __syncthreads();
    if (!sh.kept) return;
    unsigned tag = sh.tag0;
    auto valid = [&](int j, int e) { return S.act && S.c0 + e < nx && S.row0 + j < ny; };
    auto cell = [&](int j, int e) { return (size_t)(S.row0 + j) * nx + S.c0 + e; };
    // a / aP; r / aP keeps an infinite r (after an operator application an infinite value ends in NaN anyway)
    auto over_aP = [&](double a, int j, int e, bool residual = false) {
        const double d = sm[(2 * j + e) * T + S.tid];
        if (j < L::recip) {
            const double y = sm[(6 * R + 2 * j + e) * T + S.tid];
            return residual ? quotient_any(a, d, y) : quotient(a, d, y);
        }
        const bool zero = a == 0.0 && d > 0.0 && d < INFINITY;
        const double c = (zero ? d : a) / d;
        return zero ? a : c;
    };
    // a grid array's values on this thread's cells and the rows beside them
    auto load = [&](const double *g, double (&v)[R][2], double (&s)[2], double (&n)[2]) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
#pragma unroll
            for (int j = 0; j < R; j++) v[j][e] = valid(j, e) ? g[cell(j, e)] : 0.0;
            s[e] = S.row0 > 0 && valid(-1, e) ? g[cell(-1, e)] : 0.0;
            n[e] = valid(R, e) ? g[cell(R, e)] : 0.0;
        }
    };
#pragma unroll
    for (int j = 0; j < R; j++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int k = (2 * j + e) * T + S.tid;
            const bool in = valid(j, e);
            const double d = in ? A.aP[cell(j, e)] : 1.0;
            sm[k] = d;
            if (j < L::recip) sm[6 * R * T + k] = 1.0 / d;
            sm[2 * R * T + k] = in ? A.aE[cell(j, e)] : 0.0;
            sm[4 * R * T + k] = in ? A.aN[cell(j, e)] : 0.0;
        }
    S.aS0 = S.row0 > 0 && valid(0, 0) ? A.aN[cell(-1, 0)] : 0.0;
    S.aS1 = S.row0 > 0 && valid(0, 1) ? A.aN[cell(-1, 1)] : 0.0;
    // v on the thread's rows -> the operator's inputs around it (block barrier inside)
    auto share = [&](const double (&v)[R][2], double (&s)[2], double (&n)[2]) {
        if (CHEB) sb ^= 1;
        publish_block<R>(S, v, sb, ty);
        __syncthreads();
        if (ty > 1) group_rows<R>(S, sb, A.txp, ty, s, n);
    };
    // the same with the rows across block boundaries sent and received now
    auto exchange = [&](const double (&v)[R][2], double (&s)[2], double (&n)[2]) {
        tag++;
        hb ^= 1;
        send_rows<R>(A, S, v, hb, tag);
        s[0] = s[1] = n[0] = n[1] = 0.0;
        share(v, s, n);
        recv_rows<R>(A, S, hb, tag, s, n, sh.wait);
    };
    auto nothing = [&]() {};
    bool ok = true;

    double q[R][2];  // z, and A p between the two sums
    double w1[R][2]; // p; inside the Chebyshev preconditioner its search direction
    // ---- Chebyshev bounds: Lanczos from CG on D^-1 A with the right-hand side (k_est_A, k_est_B) --
    if (CHEB) {
        double s2[2], n2[2], beta = 0.0;
        load(A.rhs, q, s2, n2);
#pragma unroll
        for (int j = 0; j < R; j++) {
            r.set(j, q[j][0], q[j][1]);
            w1[j][0] = w1[j][1] = 0.0;
        }
        for (int k = 0; k < A.nsteps && ok; k++) {
#pragma unroll
            for (int j = 0; j < R; j++) {
                const double2 rj = r.get(j);
                w1[j][0] = rj.x + beta * w1[j][0];
                w1[j][1] = rj.y + beta * w1[j][1];
            }
            exchange(w1, s2, n2);
            double v[2] = {0.0, 0.0};
            apply_op<R>(S, w1, s2, n2, sb, [&](int j, double y0, double y1) {
                q[j][0] = over_aP(y0, j, 0);
                q[j][1] = over_aP(y1, j, 1);
                v[0] += w1[j][0] * q[j][0];
                v[0] += w1[j][1] * q[j][1];
                if (k == 0) {
                    v[1] += w1[j][0] * w1[j][0];
                    v[1] += w1[j][1] * w1[j][1];
                }
            });
            rb ^= 1;
            ok = all_sum<2>(
                A, sh, S.lane, S.warp, v, rb, ++tag, nothing,
                [&](double (&t)[2]) {
                    if (k == 0) ch.gamma = t[1];
                    ch.alphas[k] = ch.gamma / t[0];
                },
                [](double (&)[2]) {});
            if (!ok || k == A.nsteps - 1) break;
            const double a = ch.alphas[k];
            double w[1] = {0.0};
#pragma unroll
            for (int j = 0; j < R; j++) {
                const double2 rj = r.get(j);
                const double r0 = rj.x - a * q[j][0], r1 = rj.y - a * q[j][1];
                r.set(j, r0, r1);
                w[0] += r0 * r0;
                w[0] += r1 * r1;
            }
            rb ^= 1;
            ok = all_sum<1>(
                A, sh, S.lane, S.warp, w, rb, ++tag, nothing,
                [&](double (&t)[1]) {
                    ch.betas[k] = t[0] / ch.gamma;
                    ch.gamma = t[0];
                },
                [](double (&)[1]) {});
            beta = ch.betas[k];
        }
        __syncthreads();
        if (ok && S.warp == 0) {
            double lmin, lmax;
            cheb_bounds_warp(ch.alphas, ch.betas, A.nsteps, ch.d, ch.e, lmin, lmax);
            if (S.lane == 0) {
                ch.est_min = lmin;
                ch.est_max = lmax;
                ch.adopted = cheb_bounds_ok(lmin, lmax);
                if (ch.adopted) {
                    ch.lam_min = lmin;
                    ch.lam_max = lmax;
                }
                cheb_coefficients(ch.lam_min, ch.lam_max, A.deg, ch.ca, ch.cb);
            }
        }
        __syncthreads();
    }

    // r += f Ap, z = M^-1 r into q, partials r'z, r'r.  Jacobi: z = r / aP.  Chebyshev: k_cheb's
    // recurrence, deg - 1 operator applications.  Ends by sending z's strip-edge rows.
    double pk[CHEB ? R : 1][2];  // Chebyshev: p while w1 serves the preconditioner
    auto precond = [&](double f, double (&v)[2]) {
        if (!CHEB) {
            double v0 = 0.0, v1 = 0.0;  // the second column's partial sums
#pragma unroll
            for (int j = 0; j < R; j++) {
                const double2 rj = r.get(j);
                const double r0 = rj.x + f * q[j][0], r1 = rj.y + f * q[j][1];
                r.set(j, r0, r1);
                q[j][0] = over_aP(r0, j, 0, true);
                q[j][1] = over_aP(r1, j, 1, true);
                v[0] += r0 * q[j][0];
                v0 += r1 * q[j][1];
                v[1] += r0 * r0;
                v1 += r1 * r1;
            }
            v[0] += v0;
            v[1] += v1;
            tag++;
            hb ^= 1;
            send_rows<R>(A, S, q, hb, tag);
            return;
        }
        double rc[R][2], s2[2], n2[2], a = ch.ca[1];
#pragma unroll
        for (int j = 0; j < R; j++) {
            const double2 rj = r.get(j);
            const double rv[2] = {rj.x + f * q[j][0], rj.y + f * q[j][1]};
            r.set(j, rv[0], rv[1]);
#pragma unroll
            for (int e = 0; e < 2; e++) {
                if (L::pmode == V_REG) pk[CHEB ? j : 0][e] = w1[j][e];
                w1[j][e] = over_aP(rv[e], j, e, true);
                rc[j][e] = w1[j][e];
                q[j][e] = 0.0 + a * w1[j][e];
            }
        }
        for (int k = 2; k <= A.deg; k++) {
            exchange(w1, s2, n2);
            apply_op<R>(S, w1, s2, n2, sb, [&](int j, double y0, double y1) {
                rc[j][0] = rc[j][0] - a * over_aP(y0, j, 0);
                rc[j][1] = rc[j][1] - a * over_aP(y1, j, 1);
            });
            const double bt = ch.cb[k];
            a = ch.ca[k];
#pragma unroll
            for (int j = 0; j < R; j++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    w1[j][e] = rc[j][e] + bt * w1[j][e];
                    q[j][e] = q[j][e] + a * w1[j][e];
                }
        }
        tag++;
        hb ^= 1;
        send_rows<R>(A, S, q, hb, tag);
#pragma unroll
        for (int j = 0; j < R; j++) {
            const double2 rj = r.get(j);
            v[0] += rj.x * q[j][0];
            v[0] += rj.y * q[j][1];
            v[1] += rj.x * rj.x;
            v[1] += rj.y * rj.y;
            if (L::pmode == V_REG) w1[j][0] = pk[CHEB ? j : 0][0], w1[j][1] = pk[CHEB ? j : 0][1];
        }
    };
    double ps[2] = {0.0, 0.0}, pn[2] = {0.0, 0.0};  // p on the rows below and above the thread's
    double zs[2] = {0.0, 0.0}, zn[2] = {0.0, 0.0};  // z there
    auto recv_z = [&]() { recv_rows<R>(A, S, hb, tag - 1, zs, zn, sh.wait); };

    // ---- start: r = b - A x0, z, r'z, r'r, b'b (GROUNDED rows) ------------------------------------
    if (ok) {
        double s2[2], n2[2], v[3] = {0.0, 0.0, 0.0}, rzr[2] = {0.0, 0.0};
        load(A.x0, q, s2, n2);
        share(q, s2, n2);
        apply_op<R>(S, q, s2, n2, sb, [&](int j, double y0, double y1) {
            const double b0 = valid(j, 0) ? A.rhs[cell(j, 0)] : 0.0, b1 = valid(j, 1) ? A.rhs[cell(j, 1)] : 0.0;
            r.set(j, b0 + (-1.0) * y0, b1 + (-1.0) * y1);
            if (valid(j, 0) && A.fmask[cell(j, 0)] == M_GROUNDED) v[2] += b0 * b0;
            if (valid(j, 1) && A.fmask[cell(j, 1)] == M_GROUNDED) v[2] += b1 * b1;
        });
#pragma unroll
        for (int j = 0; j < R; j++) {
            q[j][0] = q[j][1] = 0.0;
            w1[j][0] = w1[j][1] = 0.0;
            x.set(j, 0.0, 0.0);
            if (L::pmode == V_GLOBAL) pm.set(j, 0.0, 0.0);
        }
        precond(0.0, rzr);
        v[0] = rzr[0];
        v[1] = rzr[1];
        rb ^= 1;
        ok = all_sum<3>(
            A, sh, S.lane, S.warp, v, rb, ++tag, recv_z,
            [&](double (&t)[3]) { scalars_start(sh.sc, sh.cg, t[0], t[1], t[2]); }, [](double (&)[3]) {});
    }

    // ---- iterations ----------------------------------------------------------------------------------
    CgScalars &sc = sh.sc;
    while (ok && !sc.done) {
        const double beta = sc.beta;
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (L::pmode == V_GLOBAL) {
                const double2 o = pm.get(j);
                w1[j][0] = o.x;
                w1[j][1] = o.y;
            }
            w1[j][0] = q[j][0] + beta * w1[j][0];
            w1[j][1] = q[j][1] + beta * w1[j][1];
            if (L::pmode == V_GLOBAL) pm.set(j, w1[j][0], w1[j][1]);
        }
#pragma unroll
        for (int e = 0; e < 2; e++) {
            ps[e] = zs[e] + beta * ps[e];
            pn[e] = zn[e] + beta * pn[e];
        }
        double s2[2] = {ps[0], ps[1]}, n2[2] = {pn[0], pn[1]}, v[1] = {0.0}, v1 = 0.0;
        share(w1, s2, n2);
        apply_op<R>(S, w1, s2, n2, sb, [&](int j, double y0, double y1) {
            q[j][0] = y0;
            q[j][1] = y1;
            v[0] += w1[j][0] * y0;
            v1 += w1[j][1] * y1;
        });
        v[0] += v1;
        rb ^= 1;
        ok = all_sum<1>(
            A, sh, S.lane, S.warp, v, rb, ++tag, nothing,
            [&](double (&t)[1]) {
                scalars_alpha(sc, t[0], A.eps_curv);
                wait_iteration(sh.wait, (int)sc.iter + 1);
            },
            [](double (&)[1]) {});
        if (!ok || sc.done) break;
        const double alpha = sc.alpha;
        double w[2] = {0.0, 0.0};
        precond(-alpha, w);
        rb ^= 1;
        ok = all_sum<2>(
            A, sh, S.lane, S.warp, w, rb, ++tag,
            [&]() {
                recv_z();
#pragma unroll
                for (int j = 0; j < R; j++) {
                    const double2 pj = L::pmode == V_GLOBAL ? pm.get(j) : make_double2(w1[j][0], w1[j][1]);
                    const double2 xj = x.get(j);
                    x.set(j, xj.x + alpha * pj.x, xj.y + alpha * pj.y);
                }
            },
            [&](double (&t)[2]) { scalars_beta(sc, t[0]); },
            [&](double (&t)[2]) { scalars_stop(sc, sh.cg, t[0], t[1]); });
    }

    // ---- h = x + x0 ----------------------------------------------------------------------------------
    if (S.tid == 0) sh.kept = res_end(A, sh.tag0, tag, ok);
    __syncthreads();
    if (sh.kept == kResDropped) return;
    add_to_head<R>(A, nx, ny, A.x0, A.h, [&](int j) { return x.get(j); });
    if (S.tid == 0 && sh.kept == kResSettled) {
        *A.cg = scalars_record(sc, sh.cg);
        if (CHEB) {
            A.cheb->est_min = ch.est_min;
            A.cheb->est_max = ch.est_max;
            A.cheb->adopted = ch.adopted;
            A.cheb->lam_min = ch.lam_min;
            A.cheb->lam_max = ch.lam_max;
            cheb_coefficients(ch.lam_min, ch.lam_max, kMaxChebDegree, A.cheb->calpha, A.cheb->cbeta);
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// Jacobi on at most 4096 cells (and 128 x 256): one block of 1024 threads, z, p, A p and the operator in
// shared memory, r and x in registers; nothing crosses L2 between iterations: 2.6 us an iteration at
// 16 x 16 and 5.1 at 64 x 64, where one SM's Float64 units (1.6 us) and shared memory (2.3 us) bound it;
// the general kernels take 15 (two launches and a device-side loop test).
//
// This form keeps the general kernels' sums as well: the threads take the places that k_cg_init's tiles,
// k_cg_A's row-marching blocks and k_cg_B's vector blocks give them, and partials are added along the
// same trees (block_reduce, then the last block's pass over the blocks).  The small instances of an
// ensemble, which runs those kernels, so reproduce their own single runs to the last bit; with large
// sliding coefficients a Picard loop of Krylov-default solves amplifies one rounding to 1e-6 in h within
// four timesteps.
// ---------------------------------------------------------------------------------------------------
constexpr int kTinyThreads = 1024, kTinyWarps = 32, kTinyCells = 4096;
constexpr int kTinyRows = 8;  // k_cg_A's tile height on grids this small

struct TinyArgs {
    int nx, ny;
    const double *aP, *aE, *aN, *rhs, *x0;
    double *h;
    const uint8_t *fmask;
    CgDev init;
    CgDev *cg;
    double eps_curv;
};

// The total of nb virtual blocks of W warps each, whose warp sums stand in w: block_reduce's tree over a
// block's warps, then grid_reduce's over the blocks (nb <= 32).  Every lane returns it.
template <int W>
__device__ __forceinline__ double tiny_total(const double *w, int nb, int lane) {
    double v[W];
#pragma unroll
    for (int k = 0; k < W; k++) v[k] = lane < nb ? w[lane * W + k] : 0.0;
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < o; k++) v[k] += v[k + o];
    return __shfl_sync(0xffffffffu, warp_reduce<false>(v[0]), 0);
}

__global__ void __launch_bounds__(kTinyThreads, 1) k_cg_tiny(const __grid_constant__ TinyArgs A) {
    extern __shared__ __align__(16) double sm[];
    __shared__ double wa[32 * 4], wb[2][4 * 8], wi[3][32 * 8];
    __shared__ CgDev cg;
    __shared__ CgScalars sc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nx = A.nx, ny = A.ny, n = nx * ny;
    double *Z = sm, *Pv = Z + kTinyCells, *Q = Pv + kTinyCells, *D = Q + kTinyCells, *E = D + kTinyCells,
           *N = E + kTinyCells;
    if (tid == 0) cg = A.init;
    for (int c = tid; c < n; c += kTinyThreads) {
        D[c] = A.aP[c];
        E[c] = A.aE[c];
        N[c] = A.aN[c];
        Q[c] = A.x0[c];
        Pv[c] = 0.0;
    }
    __syncthreads();
    // y = (A v)_c, subtraction order E, W, N, S
    auto apply = [&](const double *v, int ix, int iy, int c) {
        double y = D[c] * v[c];
        if (ix < nx - 1) y -= E[c] * v[c + 1];
        if (ix > 0) y -= E[c - 1] * v[c - 1];
        if (iy < ny - 1) y -= N[c] * v[c + nx];
        if (iy > 0) y -= N[c - nx] * v[c - nx];
        return y;
    };
    // ---- start, on k_cg_init's 32 x 8 tiles: r = b - A x0 (into Z), z = r / aP ---------------------
    const int tiles_x = (nx + kTX - 1) / kTX, tiles = tiles_x * ((ny + kTY - 1) / kTY);
    for (int t = warp >> 3; t < tiles; t += kTinyWarps / 8) {
        const int ix = (t % tiles_x) * kTX + lane, iy = (t / tiles_x) * kTY + (warp & 7);
        double v[3] = {0.0, 0.0, 0.0};
        if (ix < nx && iy < ny) {
            const int c = ix + iy * nx;
            const double b = A.rhs[c], r = b + (-1.0) * apply(Q, ix, iy, c), z = r / D[c];
            Z[c] = r;
            v[0] += r * z;
            v[1] += r * r;
            if (A.fmask[c] == M_GROUNDED) v[2] += b * b;
        }
#pragma unroll
        for (int k = 0; k < 3; k++) {
            v[k] = warp_reduce<false>(v[k]);
            if (lane == 0) wi[k][t * 8 + (warp & 7)] = v[k];
        }
    }
    __syncthreads();
    if (warp == 0) {
        const double rz = tiny_total<8>(wi[0], tiles, lane), rr = tiny_total<8>(wi[1], tiles, lane),
                     bb = tiny_total<8>(wi[2], tiles, lane);
        if (lane == 0) scalars_start(sc, cg, rz, rr, bb);
    }
    // ---- this thread's cells in k_cg_B's order: two pairs, and the last cell of an odd count --------
    const int nv = n / 2, nbB = (n + 1023) / 1024, i0 = tid, i1 = tid + nbB * 256;
    const bool inB = warp < nbB * 8, has0 = inB && i0 < nv, has1 = inB && i1 < nv, tail = tid == 0 && (n & 1);
    int cell[5] = {2 * i0, 2 * i0 + 1, 2 * i1, 2 * i1 + 1, n - 1};
    const bool has[5] = {has0, has0, has1, has1, tail};
    double r[5], x[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        x[k] = 0.0;
        r[k] = has[k] ? Z[cell[k]] : 0.0;
    }
    double inv[5];
#pragma unroll
    for (int k = 0; k < 5; k++) inv[k] = has[k] ? 1.0 / D[cell[k]] : 0.0;
    __syncthreads();  // every r is read: Z takes z
#pragma unroll
    for (int k = 0; k < 5; k++)
        if (has[k]) Z[cell[k]] = quotient_any(r[k], D[cell[k]], inv[k]);
    __syncthreads();
    const int nbA = (ny + kTinyRows - 1) / kTinyRows;
    while (!sc.done) {
        const double beta = sc.beta;
        for (int c = tid; c < n; c += kTinyThreads) Pv[c] = Z[c] + beta * Pv[c];
        __syncthreads();
        // A p on k_cg_A's blocks: 128 columns, 8 rows
        for (int vb = warp >> 2; vb < nbA; vb += kTinyWarps / 4) {
            const int ix = (warp & 3) * 32 + lane, y0 = vb * kTinyRows;
            double acc = 0.0;
            if (ix < nx) {
                double ps = y0 > 0 ? Pv[ix + (y0 - 1) * nx] : 0.0, ns = y0 > 0 ? N[ix + (y0 - 1) * nx] : 0.0,
                       pc = Pv[ix + y0 * nx];
#pragma unroll
                for (int j = 0; j < kTinyRows; j++) {
                    const int iy = y0 + j, c = ix + iy * nx;
                    if (iy < ny) {
                        const double pn = iy < ny - 1 ? Pv[c + nx] : 0.0, nc = N[c];
                        double y = D[c] * pc;
                        if (ix < nx - 1) y -= E[c] * Pv[c + 1];
                        if (ix > 0) y -= E[c - 1] * Pv[c - 1];
                        if (iy < ny - 1) y -= nc * pn;
                        if (iy > 0) y -= ns * ps;
                        Q[c] = y;
                        acc += pc * y;
                        ps = pc;
                        pc = pn;
                        ns = nc;
                    }
                }
            }
            acc = warp_reduce<false>(acc);
            if (lane == 0) wa[vb * 4 + (warp & 3)] = acc;
        }
        __syncthreads();
        if (warp == 0) {
            const double pAp = tiny_total<4>(wa, nbA, lane);
            if (lane == 0) scalars_alpha(sc, pAp, A.eps_curv);
        }
        __syncthreads();
        if (sc.done) break;
        const double alpha = sc.alpha;
        double v[2] = {0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 5; k++) {
            if (!has[k]) continue;
            const int c = cell[k];
            x[k] = x[k] + alpha * Pv[c];
            r[k] = r[k] + (-alpha) * Q[c];
            const double z = quotient_any(r[k], D[c], inv[k]);
            Z[c] = z;
            v[0] += r[k] * z;
            v[1] += r[k] * r[k];
        }
        if (inB) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                v[k] = warp_reduce<false>(v[k]);
                if (lane == 0) wb[k][warp] = v[k];
            }
        }
        __syncthreads();
        if (warp < 2) {
            const double rz = tiny_total<8>(wb[0], nbB, lane);
            if (warp == 0 && lane == 0) scalars_beta(sc, rz);
            if (warp == 1) {
                const double rr = tiny_total<8>(wb[1], nbB, lane);
                if (lane == 0) scalars_stop(sc, cg, rz, rr);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < 5; k++)
        if (has[k]) A.h[cell[k]] = x[k] + A.x0[cell[k]];
    if (tid == 0) *A.cg = scalars_record(sc, cg);
}

// ---------------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------------

// The geometry of a resident solve, or blocks = 0 where the grid does not fit: rows of at most 1024
// cells (two per thread), and at most 7 rows per thread on at most num_sms blocks.
// Fewer rows per thread mean less work between two exchanges, more blocks a longer exchange.  Measured
// us per iteration (plain workload, rel-res 1e-12; general kernels at the end):
//            Jacobi R = 1     2     4     7  general   Chebyshev(4) R = 1     2     4     7  general
//   100 x 90        3.8   3.9   5.0  12.2   14.4                    7.0   8.4  12.8  23.2   27.5
//   201 x 150       4.6   4.4   5.3  12.2   20.0                    8.0   9.0  13.1  23.3   28.8
//   256^2           5.1   5.0   5.3  12.1   16.2                    9.0   9.3  13.2  22.9   28.7
//   300 x 400       5.9   5.4   6.1  12.4   15.3                    9.7  10.1  13.8  23.8   31.9
//   512^2           -     5.5   6.1  12.1   18.7                    -    10.7  14.6  23.4   39.1
//   700 x 600       -     -     -    12.4   21.7                    -     -     -    24.4   46.7
//   1024^2          -     -     -    11.8   31.1                    -     -     -    26.1   83.7
// So Jacobi takes R = 2 and Chebyshev, whose iteration applies the operator four times, R = 1, and
// each the smallest larger R where those need more blocks than there are SMs.  k_cg_tiny takes the
// Jacobi solves of at most 4096 cells (3.5 us at 48 x 40, 5.1 at 64^2; general 14.1 and 15.5).
ResPlan res_plan(int nx, int ny, int num_sms, bool cheb) {
    ResPlan P;
    if (nx > 2 * kResThreads) return P;
    P.txp = (((nx + 1) / 2) + 31) / 32 * 32;
    const int groups = kResThreads / P.txp;
    auto fits = [&](int R, int most) {
        P.rows = R;
        P.ty = R > 4 ? 1 : groups;
        P.blocks = (ny + P.ty * R - 1) / (P.ty * R);
        return P.blocks <= most;
    };
    if (!cheb && nx <= 128 && ny <= 256 && nx * ny <= kTinyCells) {
        P.rows = 0;  // k_cg_tiny
        P.blocks = 1;
        return P;
    }
    for (int R : {1, 2, 4, 7})
        if ((R > 1 || cheb) && fits(R, num_sms)) return P;
    P.blocks = 0;
    return P;
}

size_t res_red_bytes(const ResPlan &P) { return (size_t)2 * P.blocks * 4 * sizeof(uint4); }
size_t res_vec_bytes(const ResPlan &P) {
    return P.rows >= 4 ? (size_t)3 * P.blocks * kResThreads * P.rows * sizeof(double2) : 0;
}
size_t res_halo_bytes(const ResPlan &P) { return (size_t)2 * P.blocks * 2 * (2 * P.txp) * sizeof(uint4); }

// A cooperative launch: the blocks run together, or not at all.  On a part of the device too small for them
// (a green context, an MPS share) it is refused, and the general kernels serve.
int res_cooperative(Ctx *c, const void *kernel, int blocks, void *args, size_t smem, const char *what) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return check_cuda(c, e, what);
    void *list[] = {args};
    e = cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(kResThreads), list, smem, c->stream);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        return kNotStarted;
    }
    c->launches++;
    return check_cuda(c, e, what);
}

template <int R, bool CHEB>
static int res_launch(Ctx *c, ResArgs &a) {
    return res_cooperative(c, (const void *)k_cg_resident<R, CHEB>, c->res[CHEB].blocks, &a, ResSmem<R, CHEB>::bytes,
                           "resident solve launch");
}

template <bool CHEB>
static int res_launch_rows(Ctx *c, ResArgs &a) {
    switch (c->res[CHEB].rows) {
    case 1: return res_launch<1, true>(c, a);  // Chebyshev only
    case 2: return res_launch<2, CHEB>(c, a);
    case 4: return res_launch<4, CHEB>(c, a);
    default: return res_launch<7, CHEB>(c, a);
    }
}

bool res_serves(const Ctx *c, const shk_cg_opts *o) {
    return o->precision == SHK_FP64 && ((o->precond == SHK_PRECOND_JACOBI && c->res[0].blocks > 0) ||
                                        (o->precond == SHK_PRECOND_CHEBYSHEV && c->res[1].blocks > 0));
}

// Tags have 31 bits: start over long before they could repeat (and after a lost solve).
int res_tags(Ctx *c) {
    if (!c->res_restart && c->host_dev->res_epoch <= (1u << 30)) return SHK_OK;
    cudaError_t e = cudaMemsetAsync(c->res_comm, 0, c->res_comm_bytes, c->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(&c->dev->res_epoch, 0, 2 * sizeof(unsigned int), c->stream);  // and res_arrived
    c->res_restart = false;
    return check_cuda(c, e, "resident solve buffers");
}

void res_waits(Ctx *c, ResComm &a) {
    a.cg = &c->dev->cg;
    a.epoch = &c->dev->res_epoch;
    a.arrived = &c->dev->res_arrived;
    a.spin = c->res_spin;
    a.start_spin = c->res_start_spin;
    a.test_absent = c->res_test_absent;
    a.test_spin = c->res_test_spin;
    a.test_block = c->res_test_block;
    a.test_iter = c->res_test_spin < 0 ? -1 : c->res_test_iter;
}

// One solve: h = x0 + the correction; the scalars end in c->dev->cg.  Asynchronous.
int res_solve(Ctx *c, const shk_cg_opts *o, const CgDev &init, const double *x0) {
    if (int rc = res_tags(c)) return rc;
    const bool cheb = o->precond == SHK_PRECOND_CHEBYSHEV;
    if (!cheb && c->res[0].rows == 0) {  // (c->march_th is kTinyRows on every grid this small)
        TinyArgs t{c->nx, c->ny, c->aP, c->aE, c->aN, c->rhs, x0, c->st.h, c->mask8, init, &c->dev->cg,
                   DBL_EPSILON};
        constexpr int smem = 6 * kTinyCells * (int)sizeof(double);
        cudaError_t e = cudaFuncSetAttribute(k_cg_tiny, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return check_cuda(c, e, "resident solve shared memory");
        k_cg_tiny<<<1, kTinyThreads, smem, c->stream>>>(t);
        c->launches++;
        return check_launch(c, "resident solve");
    }
    ResArgs a;
    a.nx = c->nx;
    a.ny = c->ny;
    a.txp = c->res[cheb].txp;
    a.ty = c->res[cheb].ty;
    a.groups = c->res[cheb].blocks;
    a.deg = cheb ? o->cheb_degree : 0;
    a.nsteps = cheb ? o->cheb_nsteps : 0;
    a.aP = c->aP;
    a.aE = c->aE;
    a.aN = c->aN;
    a.rhs = c->rhs;
    a.x0 = x0;
    a.h = c->st.h;
    a.vec = c->res_vec;
    a.fmask = c->mask8;
    a.init = init;
    a.cheb = &c->dev->cheb;
    a.red = c->res_red;
    a.halo = c->res_halo;
    a.eps_curv = DBL_EPSILON;
    res_waits(c, a);
    return cheb ? res_launch_rows<true>(c, a) : res_launch_rows<false>(c, a);
}

} // namespace shk
