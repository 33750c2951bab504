// shk_device.cuh -- device helpers: Julia-faithful scalar functions, tile iteration and the
// deterministic last-block grid reduction.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "shk_internal.cuh"

namespace shk {

// ---- scalar semantics matching the reference (Julia) -----------------------------------------

// Julia x^n for Float64 and Integer n (Base.pow_body): n == 3 is x*x*x; n == 2 gives fl(x*x);
// other n use a compensated power-by-squaring.
__device__ __forceinline__ double jl_powi(double x, int n) {
    if (n == 0) return 1.0;
    if (n == 1) return x;
    if (n == 2) return x * x;
    if (n == 3) return x * x * x;
    double y = 1.0, xnlo = 0.0, ynlo = 0.0;
    while (n > 1) {
        if (n & 1) {
            double err = fma(y, xnlo, x * ynlo);
            double hi = x * y;
            double lo = fma(x, y, -hi);
            y = hi;
            ynlo = lo + err;
        }
        double err = x * 2.0 * xnlo;
        double hi = x * x;
        double lo = fma(x, x, -hi);
        x = hi;
        xnlo = lo + err;
        n >>= 1;
    }
    double err = fma(y, xnlo, x * ynlo);
    if (isfinite(x) && isfinite(err)) return fma(x, y, fma(y, xnlo, x * ynlo));
    return x * y;
}

// pow with the reference's canonical_exponent dispatch (src/model_parameters.jl:122-134).
__device__ __forceinline__ double jl_pow(double x, double e, int e_int) {
    return e_int >= 0 ? jl_powi(x, e_int) : pow(x, e);
}

__device__ __forceinline__ double jl_max(double a, double b) {
    return (isnan(a) || isnan(b)) ? __longlong_as_double(0x7ff8000000000000LL) : (a > b ? a : b);
}
__device__ __forceinline__ double jl_min(double a, double b) {
    return (isnan(a) || isnan(b)) ? __longlong_as_double(0x7ff8000000000000LL) : (a < b ? a : b);
}
__device__ __forceinline__ double jl_sign(double x) { return x > 0 ? 1.0 : (x < 0 ? -1.0 : x); }
__device__ __forceinline__ double jl_clamp(double x, double lo, double hi) {
    return x > hi ? hi : (x < lo ? lo : x);
}

__device__ __forceinline__ bool is_dirichlet(uint8_t m) { return m == M_OCEAN || m == M_LAND; }

// a / d from the stored reciprocal y = RN(1 / d): a y, its remainder by one fused operation, and one
// correction (Markstein, IBM J. Res. Dev. 34, 1990).  3 operations where the divide takes about 20, and
// no slow path for a = 0 (fixed-head rows, cells beyond the grid), which every warp holding one such
// cell otherwise runs through; it agreed with the divide in every one of 4e9 quotients tried.
// An infinite a gives NaN; quotient_any gives the divide's infinity.
__device__ __forceinline__ double quotient(double a, double d, double y) {
    const double t = a * y;
    return fma(fma(-d, t, a), y, t);
}
__device__ __forceinline__ double quotient_any(double a, double d, double y) {
    const double t = a * y, c = fma(fma(-d, t, a), y, t);
    return (__double2hiint(t) & 0x7ff00000) == 0x7ff00000 ? t : c;  // infinite or NaN: t
}

// ---- tiles -------------------------------------------------------------------------------------

struct Tiles {
    int nx, ny, tiles_x, ntiles;
    __device__ __forceinline__ Tiles(int nx_, int ny_) : nx(nx_), ny(ny_) {
        tiles_x = (nx + kTX - 1) / kTX;
        ntiles = tiles_x * ((ny + kTY - 1) / kTY);
    }
    __device__ __forceinline__ void cell(int t, int &ix, int &iy) const {
        int tx = t % tiles_x, ty = t / tiles_x;
        ix = tx * kTX + (int)(threadIdx.x % kTX);
        iy = ty * kTY + (int)(threadIdx.x / kTX);
    }
};

// ---- reductions -----------------------------------------------------------------------------

template <bool MAX>
__device__ __forceinline__ double red_op(double a, double b) {
    if (MAX) return jl_max(a, b);
    return a + b;
}

template <bool MAX>
__device__ __forceinline__ double warp_reduce(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = red_op<MAX>(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Block-reduce NV values; result valid in thread 0.  Deterministic order.
template <int NV, bool MAX>
__device__ __forceinline__ void block_reduce(double (&v)[NV]) {
    __shared__ double sh[NV][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = warp_reduce<MAX>(v[k]);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) sh[k][warp] = v[k];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double t = lane < nwarps ? sh[k][lane] : 0.0;
            v[k] = warp_reduce<MAX>(t);
        }
    }
    __syncthreads();
}

// A block's place among the blocks that work on one instance: the single-instance kernels use
// their whole grid; the ensemble kernels give each instance a contiguous range of one grid.
struct Blk {
    int id, n;
};
__device__ __forceinline__ Blk grid_blk() { return Blk{(int)blockIdx.x, (int)gridDim.x}; }

// Grid reduction without inter-block waiting over the B.n blocks of one instance.  Returns true in
// exactly one block (the last to arrive); there, thread 0 holds the totals in out[] (other threads:
// unspecified).
template <int NV, bool MAX>
__device__ __forceinline__ bool grid_reduce(Blk B, double (&v)[NV], double *partials, unsigned int *counter,
                                            double (&out)[NV]) {
    __shared__ int am_last;
    block_reduce<NV, MAX>(v);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) partials[(size_t)k * B.n + B.id] = v[k];
        __threadfence();
        unsigned int prev = atomicAdd(counter, 1u);
        am_last = (prev == (unsigned int)B.n - 1);
    }
    __syncthreads();
    if (!am_last) return false;
    __threadfence();
    double acc[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) {
        acc[k] = 0.0;
        for (int i = threadIdx.x; i < B.n; i += blockDim.x)
            acc[k] = red_op<MAX>(acc[k], __ldcg(&partials[(size_t)k * B.n + i]));
    }
    block_reduce<NV, MAX>(acc);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) out[k] = acc[k];
        *counter = 0u;
        __threadfence();
    }
    return true;
}

template <int NV, bool MAX>
__device__ __forceinline__ bool grid_reduce(double (&v)[NV], double *partials, unsigned int *counter,
                                            double (&out)[NV]) {
    return grid_reduce<NV, MAX>(grid_blk(), v, partials, counter, out);
}

// ---------------------------------------------------------------------------------------------
// Per-block reads of the device-side CG scalars.  Thread (0,0) reads them and shares them through
// shared memory, so a launch sends one request per block to the scalars' L2 line instead of one
// per warp (a hot spot that cost more than the data traffic of the small level kernels).  Every
// thread of the block must call these, before any early return.
// ---------------------------------------------------------------------------------------------
struct CgView {
    int done, first;
    double alpha, beta, alpha_prev;
};

__device__ __forceinline__ CgView block_cg_view(const CgDev *cg) {
    __shared__ CgView v;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        v.done = *(const volatile int *)&cg->done;
        v.first = cg->first;
        v.alpha = cg->alpha;
        v.beta = cg->beta;
        v.alpha_prev = cg->alpha_prev;
    }
    __syncthreads();
    return v;
}

__device__ __forceinline__ bool block_cg_done(const int *done) {
    __shared__ int d;
    if (threadIdx.x == 0 && threadIdx.y == 0) d = done ? *(const volatile int *)done : 0;
    __syncthreads();
    return d != 0;
}

// ---------------------------------------------------------------------------------------------
// Ensemble kernels: the block's instance descriptor, copied to shared memory once per block, and
// the block's place among that instance's blocks of kernel family FAM.
// ---------------------------------------------------------------------------------------------
static_assert(sizeof(EnsInst) % 8 == 0, "EnsInst is copied in 8-byte words");
__device__ __forceinline__ Blk ens_stage(EnsInst &dst, const EnsInst *E, const int *b2i, int fam) {
    const long long *src = reinterpret_cast<const long long *>(&E[b2i[blockIdx.x]]);
    long long *d = reinterpret_cast<long long *>(&dst);
    for (int k = threadIdx.x; k < (int)(sizeof(EnsInst) / 8); k += blockDim.x) d[k] = src[k];
    __syncthreads();
    return Blk{(int)blockIdx.x - dst.blk0[fam], dst.nblk[fam]};
}

// ---------------------------------------------------------------------------------------------
// Scalar updates (run by thread 0 of the last block)
// ---------------------------------------------------------------------------------------------
static __device__ void cg_init_finish(CgDev *cg, double rz, double rr, double bb) {
    if (cg->cont) {
        // Residual replacement: keep the previous search direction, p = z + beta p with
        // beta = r'z (replaced residual) / r'z (last recursive residual).
        const double beta = rz / cg->rz_last;
        if (isfinite(beta) && beta >= 0) {
            cg->beta = beta;
            cg->pNorm2 = rz + beta * beta * cg->pNorm2;
            cg->first = 0;
        } else {
            cg->first = 1;
            cg->beta = 0.0;
            cg->pNorm2 = rz;
        }
    } else {
        cg->first = 1;
        cg->beta = 0.0;
        cg->pNorm2 = rz;
    }
    cg->gamma = rz;
    cg->rz_last = rz;
    const double rn = sqrt(rz);
    cg->rr = sqrt(rr);
    cg->bnorm = sqrt(bb);
    cg->rnorm0 = cg->stop_rule == SHK_STOP_KRYLOV ? rn : cg->rr;
    cg->rnorm = cg->rnorm0;
    cg->eps_stop = cg->atol + cg->rtol * rn;
    cg->iter = 0;
    if (isnan(rz) || isnan(rr)) {
        cg->done = 1;
        cg->status = SHK_BREAKDOWN;
    } else if (rz == 0.0) {
        cg->done = 1;
        cg->status = SHK_OK;
    } else {
        bool solved = cg->stop_rule == SHK_STOP_KRYLOV ? (rn <= cg->eps_stop) : (cg->rr <= cg->rtol * cg->bnorm);
        if (solved) {
            cg->done = 1;
            cg->status = SHK_OK;
        } else if (cg->iter >= cg->itmax) {
            cg->done = 1;
            cg->status = SHK_NOT_CONVERGED;
        } else {
            cg->done = 0;
        }
    }
}

static __device__ void cg_iter_finish(CgDev *cg, double rz, double rr) {
    const double rn = sqrt(rz), rrn = sqrt(rr);
    cg->rz_last = rz;
    cg->rr = rrn;
    bool solved;
    if (cg->stop_rule == SHK_STOP_KRYLOV) solved = (rn <= cg->eps_stop) || (rn + 1.0 <= 1.0);
    else solved = rrn <= cg->rtol * cg->bnorm;
    cg->rnorm = cg->stop_rule == SHK_STOP_KRYLOV ? rn : rrn;
    if (!solved) {
        double beta = rz / cg->gamma;
        cg->pNorm2 = rz + beta * beta * cg->pNorm2;
        cg->gamma = rz;
        cg->beta = beta;
        cg->first = 0;
    }
    cg->iter += 1;
    if (isnan(rz) || isnan(rr)) {
        cg->done = 1;
        cg->status = SHK_BREAKDOWN;
    } else if (solved) {
        cg->done = 1;
        cg->status = SHK_OK;
    } else if (cg->iter >= cg->itmax) {
        cg->done = 1;
        cg->status = SHK_NOT_CONVERGED;
    }
}

// Work queued behind a solve whose outcome the host has not read: a solve that failed (a wait that ran out,
// a loop that reached its bound) leaves the head and the fields as they were.  after = nullptr: no such solve.
static __device__ __forceinline__ bool cg_ended(const CgDev *after) { return !after || (after->done && !after->fault); }

// Programmatic dependent launch.  The kernels of an iteration are a chain of launches of a few us each; a
// kernel launched by launch_after starts while the previous one of its stream still runs, as soon as all of
// that one's blocks run, and waits here until it has completed and its writes are visible.  Every block of
// such a kernel calls after_previous before it reads what an earlier kernel of the chain wrote, before it
// writes anything and before it leaves (so the chain's order is kept from end to end); only data that no
// kernel of the chain writes may be read earlier.  (What the chain writes is not read through const
// __restrict__ pointers in such a kernel: those loads may be moved up.)  `early` = false: an ordinary launch.
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    next_may_start();
}

template <typename T>
struct Same {
    using type = T;
};
template <typename... P>
static inline cudaError_t launch_after(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                       typename Same<P>::type... a) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = early;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a...);
}

} // namespace shk
