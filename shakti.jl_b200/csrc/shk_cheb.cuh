// shk_cheb.cuh -- the scalar parts of the Chebyshev preconditioner that more than one kernel runs.
#pragma once

#include <float.h>

#include "shk_internal.cuh"

namespace shk {

// Per-step coefficients 1..deg from the bounds (src/preconditioner.jl:241-263).
static __device__ void cheb_coefficients(double lmin, double lmax, int deg, double *ca, double *cb) {
    const double d_mid = (lmax + lmin) / 2;
    const double c_rad = (lmax - lmin) / 2;
    double alpha = 1.0 / d_mid;
    ca[1] = alpha;
    cb[1] = 0.0;
    double alpha_prev = alpha;
    for (int k = 2; k <= deg; k++) {
        double t = c_rad * alpha_prev / 2;
        double beta = t * t;
        alpha = 1.0 / (d_mid - beta / alpha_prev);
        ca[k] = alpha;
        cb[k] = beta;
        alpha_prev = alpha;
    }
}

// Sturm count of eigenvalues below x for SymTridiagonal(d, e).
static __device__ int cheb_sturm(int m, const double *d, const double *e, double x) {
    int cnt = 0;
    double q = d[0] - x;
    if (q < 0) cnt++;
    for (int i = 1; i < m; i++) {
        if (q == 0) q = DBL_EPSILON * (fabs(e[i - 1]) + DBL_MIN);
        q = d[i] - x - e[i - 1] * e[i - 1] / q;
        if (q < 0) cnt++;
    }
    return cnt;
}

// Validity test of update_chebyshev_bounds! (src/preconditioner.jl:219-230).
static __device__ bool cheb_bounds_ok(double lmin, double lmax) {
    return isfinite(lmin) && isfinite(lmax) && lmin > 0 && lmax > lmin;
}

// estimate_eigenvalue_bounds' tail (src/preconditioner.jl:115-133) from the Lanczos coefficients of m
// steps, by one whole warp; d, e: shared scratch of m values.  LAPACK's eigvals(SymTridiagonal) is
// replaced by Sturm counts for the two extreme eigenvalues (the only ones used): each half of the warp
// sections its bracket at 16 points at once, down to adjacent doubles.  (One thread's bisection took
// 180 us of every Chebyshev solve, the serial chain of 2 x 53 Sturm counts with a divide per step.)
static __device__ void cheb_bounds_warp(const double *alphas, const double *betas, int m, double *d, double *e,
                                        double &lmin, double &lmax) {
    const int lane = threadIdx.x & 31;
    for (int k = lane; k < m; k += 32) {
        d[k] = k == 0 ? 1 / alphas[0] : 1 / alphas[k] + betas[k - 1] / alphas[k - 1];
        if (k < m - 1) e[k] = sqrt(betas[k]) / alphas[k];
    }
    __syncwarp();
    bool finite = true;
    double lo = INFINITY, hi = -INFINITY;
    for (int i = 0; i < m; i++) {
        finite = finite && isfinite(d[i]) && (i + 1 >= m || isfinite(e[i]));
        const double rad = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < m ? fabs(e[i]) : 0.0);
        lo = fmin(lo, d[i] - rad);
        hi = fmax(hi, d[i] + rad);
    }
    lmin = lmax = __longlong_as_double(0x7ff8000000000000LL);
    if (!finite) return;
    const double span = fmax(fabs(lo), fabs(hi));
    double a = lo - (DBL_EPSILON * span + DBL_MIN), b = hi + (DBL_EPSILON * span + DBL_MIN);
    const int half = lane >> 4, l = lane & 15, target = half ? m : 1;
    for (int it = 0; it < 64; it++) {
        const double x = a + (b - a) * ((l + 1) / 17.0);
        const bool above = x >= b || (x > a && cheb_sturm(m, d, e, x) >= target);
        const unsigned bal = (__ballot_sync(0xffffffffu, above) >> (16 * half)) & 0xffffu;
        const int f = bal ? __ffs(bal) - 1 : 16;  // the first point above the eigenvalue
        const double xa = __shfl_sync(0xffffffffu, x, 16 * half + (f > 0 ? f - 1 : 0));
        const double xb = __shfl_sync(0xffffffffu, x, 16 * half + (f < 16 ? f : 15));
        const double na = f > 0 ? fmax(a, xa) : a, nb = f < 16 ? fmin(b, xb) : b;
        const bool moved = na != a || nb != b;
        a = na;
        b = nb;
        if (!__any_sync(0xffffffffu, moved)) break;
    }
    const double root = 0.5 * (a + b);
    lmin = __shfl_sync(0xffffffffu, root, 0) * 0.9;
    lmax = __shfl_sync(0xffffffffu, root, 16) * 1.1;
}

} // namespace shk
