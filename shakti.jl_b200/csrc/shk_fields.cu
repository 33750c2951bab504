// shk_fields.cu -- point-wise and stencil field kernels of libshakti_b200:
//   set_initial_conditions!, update_MFLS! assembly, the fused Picard tail, relax_h!, step_b!.
//
// Every value is produced with the reference's formula and evaluation order (the library is
// compiled with --fmad=false, so no a*b+c is contracted), which makes these kernels bit-identical
// to the reference's unfused kernels except for x^(1/n) (cbrt for n = 3, pow otherwise), which may
// differ from Julia's x^(1/n) in the last bit.  Fusion never changes a value: a face quantity needed by two cells is
// computed once from the same operands and shared.
#include <cuda_runtime.h>
#include <float.h>

#include <algorithm>

#include "shk_device.cuh"

namespace shk {

#define CI(ix, iy) ((size_t)(ix) + (size_t)(iy) * (size_t)nx)
#define XI(ix, iy) ((size_t)(ix) + (size_t)(iy) * (size_t)(nx + 1))
#define YI(ix, iy) ((size_t)(ix) + (size_t)(iy) * (size_t)nx)

// ---------------------------------------------------------------------------------------------
// Mask
// ---------------------------------------------------------------------------------------------

__global__ void k_mask8(int n, const double *__restrict__ mask, uint8_t *__restrict__ m8) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double m = mask[i];
        uint8_t c = M_UNKNOWN;
        if (m == 0.0) c = M_GROUNDED;
        else if (m == 1.0) c = M_OCEAN;
        else if (m == 2.0) c = M_LAND;
        else if (m == 3.0) c = M_OTHER;
        m8[i] = c;
    }
}

// compute_valid_x/y_kernel! (src/mask.jl:62-84) and apply_mask_to_sliding_x/y_kernel!
// (src/mask.jl:117-136): one thread per face.
__global__ void k_face_masks_and_sliding(int nx, int ny, const uint8_t *__restrict__ m8,
                                         double *valid_x, double *valid_y, double *ub_x, double *ub_y) {
    const long long nxf = (long long)(nx + 1) * ny, nyf = (long long)nx * (ny + 1);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nxf + nyf;
         i += (long long)gridDim.x * blockDim.x) {
        if (i < nxf) {
            int f = (int)(i % (nx + 1)), iy = (int)(i / (nx + 1));
            bool interior = f > 0 && f < nx;
            double v = 1.0;
            bool both_grounded = false;
            if (interior) {
                uint8_t a = m8[CI(f - 1, iy)], b = m8[CI(f, iy)];
                v = (a != M_OTHER && b != M_OTHER) ? 1.0 : 0.0;
                both_grounded = a == M_GROUNDED && b == M_GROUNDED;
            }
            valid_x[i] = v;
            if (!interior || !both_grounded) ub_x[i] = 0.0;
        } else {
            long long j = i - nxf;
            int ix = (int)(j % nx), f = (int)(j / nx);
            bool interior = f > 0 && f < ny;
            double v = 1.0;
            bool both_grounded = false;
            if (interior) {
                uint8_t a = m8[CI(ix, f - 1)], b = m8[CI(ix, f)];
                v = (a != M_OTHER && b != M_OTHER) ? 1.0 : 0.0;
                both_grounded = a == M_GROUNDED && b == M_GROUNDED;
            }
            valid_y[j] = v;
            if (!interior || !both_grounded) ub_y[j] = 0.0;
        }
    }
}

// ---------------------------------------------------------------------------------------------
// set_initial_conditions! (src/initial_conditions.jl:14-125), centre steps in reference order.
// ---------------------------------------------------------------------------------------------
__global__ void k_init_center(int n, Params P, shk_state s, const uint8_t *__restrict__ m8) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint8_t m = m8[i];
        const double lambda_coeff = 1.5;
        s.lambda[i] = lambda_coeff * s.A_visc[i];
        double b = s.b[i];
        b = (s.mask[i] != 0.0) ? 0.0 : b; // ifelse(mask != GROUNDED, 0, b)
        s.b[i] = b;
        double H = s.zs[i] - (s.zb[i] + b); // compute_H!
        s.H[i] = H;
        if (P.br != 0.0) s.beta[i] = jl_max(0.0, (P.br - b) / P.lr); // compute_beta!
        double po = P.rho_i * P.g * H; // compute_po!
        s.po[i] = po;
        double pw = po / 2;
        if (m == M_OCEAN) pw = P.p_atm - P.rho_sw * P.g * jl_min(s.zb[i], 0.0);
        else if (m == M_LAND || m == M_OTHER) pw = P.p_atm;
        s.pw[i] = pw;
        // compute_N! then compute_h!
        double d = po - pw;
        s.N[i] = (m == M_GROUNDED) ? d : copysign(0.0, d);
        s.h[i] = pw / (P.rho_w * P.g) + s.zb[i];
    }
}

// compute_abs_ub! (src/static_fields.jl:59-66)
__global__ void k_abs_ub(int nx, int ny, shk_state s) {
    const int n = nx * ny;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int ix = i % nx, iy = i / nx;
        double ubx_c = (s.ub_x[XI(ix, iy)] + s.ub_x[XI(ix + 1, iy)]) / 2;
        double uby_c = (s.ub_y[YI(ix, iy)] + s.ub_y[YI(ix, iy + 1)]) / 2;
        s.abs_ub[i] = sqrt(ubx_c * ubx_c + uby_c * uby_c);
    }
}

// compute_dpwdx!/dpwdy!, compute_dhdx!/dhdy!, compute_b_x!/b_y! (initial-condition order; the
// gradient edge faces are never written).
__global__ void k_init_faces(int nx, int ny, Params P, shk_state s) {
    const long long nxf = (long long)(nx + 1) * ny, nyf = (long long)nx * (ny + 1);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nxf + nyf;
         i += (long long)gridDim.x * blockDim.x) {
        if (i < nxf) {
            int f = (int)(i % (nx + 1)), iy = (int)(i / (nx + 1));
            if (f > 0 && f < nx) {
                size_t a = CI(f - 1, iy), b = CI(f, iy);
                s.dpwdx[i] = ((s.pw[b] - s.pw[a]) / P.dx) * s.valid_x[i];
                s.dhdx[i] = ((s.h[b] - s.h[a]) / P.dx) * s.valid_x[i];
                s.b_x[i] = (s.b[b] + s.b[a]) / 2;
            } else {
                s.b_x[i] = s.b[CI(f == 0 ? 0 : nx - 1, iy)];
            }
        } else {
            long long j = i - nxf;
            int ix = (int)(j % nx), f = (int)(j / nx);
            if (f > 0 && f < ny) {
                size_t a = CI(ix, f - 1), b = CI(ix, f);
                s.dpwdy[j] = ((s.pw[b] - s.pw[a]) / P.dy) * s.valid_y[j];
                s.dhdy[j] = ((s.h[b] - s.h[a]) / P.dy) * s.valid_y[j];
                s.b_y[j] = (s.b[b] + s.b[a]) / 2;
            } else {
                s.b_y[j] = s.b[CI(ix, f == 0 ? 0 : ny - 1)];
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Face physics shared by the tail: q/Re (src/water_flux.jl:192-208) and taub (src/sliding_law.jl)
// ---------------------------------------------------------------------------------------------
struct FaceOut {
    double dh, dpw, q, re, taub, ub;
};

__device__ __forceinline__ void q_re(const Params &P, double bf, double grad, double &q, double &re) {
    double G = fabs(grad);
    double D = quotient_any(bf * bf * bf * P.g * G, P.nu2x12, P.nu2x12_inv);
    double R = 2 * D / (1 + sqrt(1 + 4 * P.omega * D));
    re = R;
    q = -jl_sign(grad) * P.nu * R;
}

// One face of any sliding law.  Nf/lf/abs_v already staggered; Cf the face coefficient.
__device__ __forceinline__ double taub_face(const Params &P, const Sliding &L, double Nf, double lf,
                                            double abs_v, double ub, double Cf) {
    if (L.kind == SHK_SLIDING_LINEAR) return Cf * Nf * ub;
    if (!(abs_v > 0)) return 0.0;
    double denom = (L.kind == SHK_SLIDING_REG_COULOMB_V0) ? L.v0 : jl_pow(fabs(Nf), P.n, P.n_int) * lf;
    // no sliding across this face: the drag is 0 (with its sign) where the root below is finite, which a
    // ratio in [0, 1] gives (a negative denominator, from v0 < 0 or lambda < 0, may give NaN or infinity)
    if (ub == 0.0 && abs_v < INFINITY && denom >= 0) return Nf * Cf * ub;
    // x^(1/n): for n = 3, cbrt (a fraction of pow's cost; it differs from pow(x, 1/3.0) by at most
    // about an ulp, within the tolerance the parity tests hold the pow-dependent fields to)
    const double ratio = abs_v / (abs_v + denom);
    return Nf * Cf * (P.root3 ? cbrt(ratio) : jl_pow(ratio, P.inv_n, -1)) * (ub / abs_v);
}

// Cell-centred quantities needed by faces.
struct CellQ {
    double h, pw, N, lam, aub;
};

// What a cell's CellQ is formed from, as loaded: h, zb, po (FROM_H) or h, pw, N.
struct CellRaw {
    double a, b, c, lam, aub;
    uint8_t m;
};
template <bool FROM_H>
__device__ __forceinline__ CellRaw load_cell(const shk_state &s, const uint8_t *m8, unsigned c) {
    CellRaw r;
    r.a = s.h[c];
    r.b = FROM_H ? s.zb[c] : s.pw[c];
    r.c = FROM_H ? s.po[c] : s.N[c];
    r.lam = s.lambda[c];
    r.aub = s.abs_ub[c];
    r.m = FROM_H ? m8[c] : 0;
    return r;
}
template <bool FROM_H>
__device__ __forceinline__ CellQ make_cell(const Params &P, const CellRaw &r) {
    CellQ q;
    q.h = r.a;
    if (FROM_H) {
        q.pw = P.rho_w * P.g * (q.h - r.b);
        const double d = r.c - q.pw;
        q.N = (r.m == M_GROUNDED) ? d : copysign(0.0, d);
    } else {
        q.pw = r.b;
        q.N = r.c;
    }
    q.lam = r.lam;
    q.aub = r.aub;
    return q;
}

// A face's own inputs.
struct FaceRaw {
    double valid, b, ub;
};
// Where a law keeps its face coefficients, or the prescribed drag (nullptr: one coefficient for all faces).
// They are requested with a row's first loads: fetched where the drag is formed, after the square root, they
// were one more wait per face (3000 x 3000, v0 law: 659 us; 769 so, and 715 before the warps marched).
template <int DIR>
__device__ __forceinline__ const double *face_coef(const Sliding &L, const shk_state &s) {
    if (L.kind == SHK_SLIDING_PRESCRIBED) return DIR == 0 ? s.taub_x : s.taub_y;
    return L.kind == SHK_SLIDING_REG_COULOMB ? nullptr : (DIR == 0 ? L.Cx : L.Cy);
}

// x- (DIR 0) or y-face (DIR 1) between cells a (west/south) and b (east/north); a or b may be absent
// at the domain edge (edge face: gradients read from memory, taub uses the one adjacent cell).
template <bool FROM_H, int DIR>
__device__ __forceinline__ FaceOut face(const Params &P, const Sliding &L, const shk_state &s, unsigned fi, bool interior, const CellQ &a, const CellQ &b, const CellQ &edge_cell,
                                        const FaceRaw &r, double Cf) {
    FaceOut o;
    if (interior && FROM_H) {
        const double dd = DIR == 0 ? P.dx : P.dy, inv = DIR == 0 ? P.dx_inv : P.dy_inv;
        o.dh = quotient_any(b.h - a.h, dd, inv) * r.valid;
        o.dpw = quotient_any(b.pw - a.pw, dd, inv) * r.valid;
    } else {
        o.dh = (DIR == 0 ? s.dhdx : s.dhdy)[fi];
        o.dpw = (DIR == 0 ? s.dpwdx : s.dpwdy)[fi];
    }
    q_re(P, r.b, o.dh, o.q, o.re);
    o.ub = r.ub;
    if (L.kind == SHK_SLIDING_PRESCRIBED) {
        o.taub = Cf;
    } else {
        double Nf, lf, av;
        if (interior) {
            Nf = (b.N + a.N) / 2;
            lf = (b.lam + a.lam) / 2;
            av = (b.aub + a.aub) / 2;
        } else {
            Nf = edge_cell.N;
            lf = edge_cell.lam;
            av = edge_cell.aub;
        }
        o.taub = taub_face(P, L, Nf, lf, av, o.ub, Cf);
    }
    return o;
}

// ---------------------------------------------------------------------------------------------
// Fused tail: compute_dhdxy!, compute_pw!, compute_dpwdxy!, compute_N!, compute_q_and_Re_xy!,
// compute_Re!, compute_taub_xy!, compute_mdot!, compute_K! (src/elliptic_solver.jl:193-206),
// plus the Picard check maxima max|h - h_prev| and max|h| (src/elliptic_solver.jl:162-163).
// FROM_H = false is the initial-condition variant: pw, N and the gradients are taken as set.
//
// A warp marches up a strip of 30 columns (lanes 1..30; lanes 0 and 31 hold the columns beside it).  Row by
// row it forms the row's west faces from its cells (a lane's west cell by shuffle; its east face is the
// next lane's west face) and the north faces from the row above, which the next row takes as its south
// faces: no shared memory, no block barrier, every face computed once but for the strips' edges (6 %,
// and one row of faces per strip).  The next row's 14 inputs are requested before the current row is
// computed, so 16 warps per SM keep 45 KB of loads in flight.  The strips' height makes one wave of the
// resident warps.
// 257 B per cell: 344 us at 2501 x 1803 and 1240 us at 4096^2 (53 % of the copy rate), where the form
// before it (32 x 8 tiles, faces through shared memory, three waits per tile) took 389 and 1302.  Bound
// by latency: about 1000 instructions a row, a fifth of them Float64, in chains that the branches
// inside divides, square roots and the cube root keep from overlapping, on 16 warps an SM (12 warps:
// 399 us at 2501 x 1803; 20 with spills: 491; without the prefetch and 24 warps: 367).
// ---------------------------------------------------------------------------------------------
constexpr int kTailCols = 30;  // output columns of a warp

// What a cell needs of a face.
struct FaceSums {
    double re, ut, qd, qp;  // Re, ub*taub, q*dh, q*dpw
};
__device__ __forceinline__ FaceSums face_sums(const FaceOut &o) {
    return FaceSums{o.re, o.ub * o.taub, o.q * o.dh, o.q * o.dpw};
}

// COEF: the law may have face coefficients (false: the launch knows that it has one for all faces).
template <bool FROM_H, bool CHECK, bool COEF>
__device__ __forceinline__ void tail_body(Blk B, int nx, int ny, const Params &P, const Sliding &L,
                                          const shk_state &s, const uint8_t *__restrict__ m8,
                                          const double *__restrict__ h_prev, double *partials, unsigned int *counter,
                                          PicDev *pic) {
    const int lane = threadIdx.x & 31, warps = B.n * (kTailThreads / 32);
    const int nsx = (nx + kTailCols - 1) / kTailCols, per = max(1, warps / nsx), th = (ny + per - 1) / per,
              strips = nsx * ((ny + th - 1) / th);
    const double *const cx = COEF ? face_coef<0>(L, s) : nullptr, *const cy = COEF ? face_coef<1>(L, s) : nullptr;
    double red[2] = {0.0, 0.0};
    for (int st = B.id * (kTailThreads / 32) + (threadIdx.x >> 5); st < strips; st += warps) {
        const int ix = (st % nsx) * kTailCols - 1 + lane, y0 = (st / nsx) * th, y1 = min(y0 + th, ny);
        const bool own = lane >= 1 && lane <= kTailCols && ix < nx;
        const bool xown = own || (lane >= 1 && ix == nx);   // writes its west face (ix = nx: the domain's east edge)
        const bool xint = ix > 0 && ix < nx;
        // Lanes beyond the grid read the nearest cell and face, rows beyond it the last row: every load
        // is in bounds without a test, and what those lanes compute is not written.
        const unsigned kx = min(max(ix, 0), nx - 1), kf = min(max(ix, 0), nx);
        unsigned c = (unsigned)y0 * nx + kx, fx = (unsigned)y0 * (nx + 1) + kf;  // row iy's cell, west face; south face c
        auto cell = [&](unsigned k) { return load_cell<FROM_H>(s, m8, k); };
        auto yface = [&](unsigned k) { return FaceRaw{s.valid_y[k], s.b_y[k], s.ub_y[k]}; };
        auto xface = [&](unsigned k) { return FaceRaw{s.valid_x[k], s.b_x[k], s.ub_x[k]}; };
        auto put_y = [&](unsigned fi, bool interior, const FaceOut &o) {
            if (interior && FROM_H) {
                s.dhdy[fi] = o.dh;
                s.dpwdy[fi] = o.dpw;
            }
            s.q_y[fi] = o.q;
            s.Re_y[fi] = o.re;
            if (L.kind != SHK_SLIDING_PRESCRIBED) s.taub_y[fi] = o.taub;
        };
        // the strip's first row and the faces below it
        const CellRaw below = cell(y0 > 0 ? c - nx : c), first = cell(c);
        const FaceRaw fs = yface(c);
        CellRaw next_r = cell(y0 + 1 < ny ? c + nx : c);
        FaceRaw north_r = yface(c + nx), west_r = xface(fx);
        CellQ cur = make_cell<FROM_H>(P, first);
        FaceSums S;
        {
            const CellQ q = make_cell<FROM_H>(P, below);
            const FaceOut o = face<FROM_H, 1>(P, L, s, c, y0 > 0, q, cur, cur, fs, cy ? cy[c] : L.C);
            if (own) put_y(c, y0 > 0, o);
            S = face_sums(o);
        }
        for (int iy = y0; iy < y1; iy++, c += nx, fx += nx + 1) {
            const double Cn = cy ? cy[c + nx] : L.C, Cw = cx ? cx[fx] : L.C;
            const double G = s.G[c], bb = s.b[c], hp = CHECK ? h_prev[c] : 0.0;
            // the next row's inputs
            const bool more = iy + 1 < y1;
            const unsigned cn = more ? c + nx : c;
            const CellRaw next2_r = cell(iy + 2 < ny ? cn + nx : cn);
            const FaceRaw north2_r = yface(cn + nx), west2_r = xface(more ? fx + nx + 1 : fx);
            const CellQ nxt = make_cell<FROM_H>(P, next_r);
            // north face
            const bool nint = iy + 1 < ny;
            const FaceOut on = face<FROM_H, 1>(P, L, s, c + nx, nint, cur, nxt, cur, north_r, Cn);
            if (own && (more || !nint)) put_y(c + nx, nint, on);
            const FaceSums Nf = face_sums(on);
            // west face
            CellQ w;
            w.h = __shfl_up_sync(0xffffffffu, cur.h, 1);
            w.pw = __shfl_up_sync(0xffffffffu, cur.pw, 1);
            w.N = __shfl_up_sync(0xffffffffu, cur.N, 1);
            w.lam = __shfl_up_sync(0xffffffffu, cur.lam, 1);
            w.aub = __shfl_up_sync(0xffffffffu, cur.aub, 1);
            const FaceOut ow = face<FROM_H, 0>(P, L, s, fx, xint, w, cur, ix > 0 ? w : cur, west_r, Cw);
            if (xown) {
                if (xint && FROM_H) {
                    s.dhdx[fx] = ow.dh;
                    s.dpwdx[fx] = ow.dpw;
                }
                s.q_x[fx] = ow.q;
                s.Re_x[fx] = ow.re;
                if (L.kind != SHK_SLIDING_PRESCRIBED) s.taub_x[fx] = ow.taub;
            }
            const FaceSums W = face_sums(ow);
            FaceSums E;
            E.re = __shfl_down_sync(0xffffffffu, W.re, 1);
            E.ut = __shfl_down_sync(0xffffffffu, W.ut, 1);
            E.qd = __shfl_down_sync(0xffffffffu, W.qd, 1);
            E.qp = __shfl_down_sync(0xffffffffu, W.qp, 1);
            if (own) {
                if (FROM_H) {
                    s.pw[c] = cur.pw;
                    s.N[c] = cur.N;
                }
                // compute_Re! (src/water_flux.jl:107-112)
                const double Re_c = (W.re + E.re + S.re + Nf.re) / 4;
                s.Re[c] = Re_c;
                // compute_mdot! (src/melt_rate.jl:106-137)
                const double sh = fabs((E.ut + W.ut) / 2 + (Nf.ut + S.ut) / 2);
                const double pot = fabs((E.qd + W.qd) / 2 + (Nf.qd + S.qd) / 2);
                s.shear[c] = sh;
                s.potential[c] = pot;
                if (P.with_sensible) {
                    const double sens = (E.qp + W.qp) / 2 + (Nf.qp + S.qp) / 2;
                    s.sensible[c] = sens;
                    s.mdot[c] = P.Linv * (G + sh + P.rho_w * P.g * pot + P.ct * P.cw * P.rho_w * sens);
                } else {
                    s.mdot[c] = P.Linv * (G + sh + P.rho_w * P.g * pot);
                }
                // compute_K! (src/water_flux.jl:221-226)
                s.K[c] = (bb * bb * bb * P.g) / (12 * P.nu * (1 + P.omega * Re_c));
                if (CHECK) {
                    red[0] = jl_max(red[0], fabs(cur.h - hp));
                    red[1] = jl_max(red[1], fabs(cur.h));
                }
            }
            S = Nf;
            cur = nxt;
            next_r = next2_r;
            north_r = north2_r;
            west_r = west2_r;
        }
    }
    if (CHECK) {
        double out[2];
        if (grid_reduce<2, true>(B, red, partials, counter, out) && threadIdx.x == 0) {
            pic->dmax = out[0];
            pic->hmax = out[1];
        }
    }
}

template <bool FROM_H, bool CHECK, bool COEF>
__global__ void __launch_bounds__(kTailThreads, kTailBlocksPerSm) k_tail(int nx, int ny, Params P, Sliding L, shk_state s,
                                                      const uint8_t *__restrict__ m8,
                                                      const double *__restrict__ h_prev, double *partials,
                                                      unsigned int *counter, PicDev *pic, const CgDev *after) {
    if (!cg_ended(after)) return;
    tail_body<FROM_H, CHECK, COEF>(grid_blk(), nx, ny, P, L, s, m8, h_prev, partials, counter, pic);
}

// ---------------------------------------------------------------------------------------------
// Assembly: update_MFLS_kernel! / update_MFLS_parabolic_kernel! (src/linear_solver.jl:438-588)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ double dirichlet_head(const Params &P, uint8_t m, double zb) {
    if (m == M_OCEAN) {
        double pw_bc = P.p_atm - P.rho_sw * P.g * jl_min(zb, 0.0);
        return pw_bc / (P.rho_w * P.g) + zb;
    }
    return P.p_atm / (P.rho_w * P.g) + zb;
}

// boundary_K_face (src/k_face_scheme.jl:52-61)
__device__ __forceinline__ double bK(int kfs, double K1, double K2, uint8_t m2) {
    if (m2 == M_OTHER) return 0.0;
    if (m2 == M_OCEAN || m2 == M_LAND) return K1;
    if (kfs == SHK_KFACE_HARMONIC) return (2 * K1 * K2) / (K1 + K2 + DBL_EPSILON);
    return (K1 + K2) / 2;
}

template <bool PARABOLIC>
__device__ __forceinline__ void assemble_body(Blk B, int nx, int ny, const Params &P, int kfs, double dt,
                                              const shk_state &s, const uint8_t *__restrict__ m8,
                                              double *__restrict__ aP, double *__restrict__ aE,
                                              double *__restrict__ aN, double *__restrict__ rhs,
                                              double *__restrict__ h_prev) {
    Tiles T(nx, ny);
    for (int t = B.id; t < T.ntiles; t += B.n) {
        int ix, iy;
        T.cell(t, ix, iy);
        if (ix >= nx || iy >= ny) continue;
        const size_t c = CI(ix, iy);
        // every input is loaded before the first branch, so that the loads are in flight together
        // (the Dirichlet and OTHER_BASIN rows use few of them)
        const bool hE = ix < nx - 1, hW = ix > 0, hN = iy < ny - 1, hS = iy > 0;
        const uint8_t m = m8[c];
        const uint8_t mE = hE ? m8[c + 1] : 0, mW = hW ? m8[c - 1] : 0, mN = hN ? m8[c + nx] : 0,
                      mS = hS ? m8[c - nx] : 0;
        const double h = s.h[c], zb = s.zb[c], K = s.K[c];
        const double KE = hE ? s.K[c + 1] : 0.0, KW = hW ? s.K[c - 1] : 0.0, KN = hN ? s.K[c + nx] : 0.0,
                     KS = hS ? s.K[c - nx] : 0.0;
        const double Nc = s.N[c], A = s.A_visc[c], b = s.b[c], mdot = s.mdot[c], beta = s.beta[c],
                     aub = s.abs_ub[c], ieb = s.ieb[c];
        if (h_prev) h_prev[c] = h;
        double oP, oE = 0.0, oN = 0.0, orhs;
        if (is_dirichlet(m)) {
            oP = 1;
            orhs = dirichlet_head(P, m, zb);
        } else if (m == M_OTHER) {
            oP = 1;
            orhs = h;
        } else {
            double eE = 0.0, eW = 0.0, eN = 0.0, eS = 0.0;
            if (hE) eE = bK(kfs, K, KE, mE) / P.dx2;
            if (hW) eW = bK(kfs, K, KW, mW) / P.dx2;
            if (hN) eN = bK(kfs, K, KN, mN) / P.dy2;
            if (hS) eS = bK(kfs, K, KS, mS) / P.dy2;
            const double Nn = jl_pow(fabs(Nc), P.nm1, P.nm1_int);
            if (PARABOLIC) oP = (eE + eW + eN + eS) + P.e_v / dt;
            else oP = (eE + eW + eN + eS) + P.n * P.rho_w * P.g * A * Nn * b;
            double drhs = 0.0;
            if (ix < nx - 1) {
                if (is_dirichlet(mE)) drhs += eE * dirichlet_head(P, mE, s.zb[c + 1]);
                else oE = eE;
            }
            if (ix > 0 && is_dirichlet(mW)) drhs += eW * dirichlet_head(P, mW, s.zb[c - 1]);
            if (iy < ny - 1) {
                if (is_dirichlet(mN)) drhs += eN * dirichlet_head(P, mN, s.zb[c + nx]);
                else oN = eN;
            }
            if (iy > 0 && is_dirichlet(mS)) drhs += eS * dirichlet_head(P, mS, s.zb[c - nx]);
            if (PARABOLIC)
                orhs = mdot * (1 / P.rho_w - 1 / P.rho_i) - beta * aub + A * Nn * Nc * b + ieb + (P.e_v / dt) * h +
                       drhs;
            else
                orhs = mdot * (1 / P.rho_w - 1 / P.rho_i) - beta * aub + A * Nn * Nc * b +
                       A * Nn * (P.n * P.rho_w * P.g * h) * b + ieb + drhs;
        }
        aP[c] = oP;
        aE[c] = oE;
        aN[c] = oN;
        rhs[c] = orhs;
    }
}

template <bool PARABOLIC>
__global__ void __launch_bounds__(kThreads, kAsmBlocksPerSm) k_assemble(int nx, int ny, Params P, int kfs, double dt,
                                                       shk_state s, const uint8_t *__restrict__ m8,
                                                       double *__restrict__ aP, double *__restrict__ aE,
                                                       double *__restrict__ aN, double *__restrict__ rhs,
                                                       double *__restrict__ h_prev) {
    assemble_body<PARABOLIC>(grid_blk(), nx, ny, P, kfs, dt, s, m8, aP, aE, aN, rhs, h_prev);
}

__global__ void k_export_mfls(int nx, int ny, const double *aP, const double *aE, const double *aN,
                              const double *rhs, double *oP, double *oE, double *oW, double *oN, double *oS,
                              double *orhs) {
    const int n = nx * ny;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int ix = i % nx, iy = i / nx;
        if (oP) oP[i] = aP[i];
        if (oE) oE[i] = aE[i];
        if (oN) oN[i] = aN[i];
        if (oW) oW[i] = ix > 0 ? aE[i - 1] : 0.0;
        if (oS) oS[i] = iy > 0 ? aN[i - nx] : 0.0;
        if (orhs) orhs[i] = rhs[i];
    }
}

// relax_h! (src/elliptic_solver.jl:42-46)
__global__ void k_relax(int n, double alpha, double *h, const double *h_prev, const CgDev *after) {
    if (!cg_ended(after)) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        h[i] = alpha * h[i] + (1 - alpha) * h_prev[i];
}

// compute_b_implicit/explicit_kernel! (src/gap_height.jl:117-135) then compute_beta! (:47-52).
template <bool IMPLICIT>
__device__ __forceinline__ void gap_b_body(Blk B, int n, const Params &P, double dt, const shk_state &s) {
    for (int i = B.id * blockDim.x + threadIdx.x; i < n; i += B.n * blockDim.x) {
        double b = s.b[i];
        if (s.mask[i] == 0.0) {
            const double Nc = s.N[i];
            const double Nn = jl_pow(fabs(Nc), P.nm1, P.nm1_int);
            double bnew;
            if (IMPLICIT)
                bnew = (b + dt * (s.mdot[i] / P.rho_i + s.beta[i] * s.abs_ub[i])) / (1 + dt * s.A_visc[i] * Nn * Nc);
            else
                bnew = b + dt * (s.mdot[i] / P.rho_i + s.beta[i] * s.abs_ub[i] - s.A_visc[i] * Nn * Nc * b);
            b = jl_clamp(bnew, P.b_min, P.b_max);
            s.b[i] = b;
        }
        if (P.br != 0.0) s.beta[i] = jl_max(0.0, (P.br - b) / P.lr);
    }
}

template <bool IMPLICIT>
__global__ void k_gap_b(int n, Params P, double dt, shk_state s, const uint8_t *__restrict__ m8) {
    gap_b_body<IMPLICIT>(grid_blk(), n, P, dt, s);
}

// compute_b_x!/compute_b_y! (src/gap_height.jl:75-108)
__device__ __forceinline__ void gap_faces_body(Blk B, int nx, int ny, const shk_state &s) {
    const long long nxf = (long long)(nx + 1) * ny, nyf = (long long)nx * (ny + 1);
    for (long long i = B.id * (long long)blockDim.x + threadIdx.x; i < nxf + nyf;
         i += (long long)B.n * blockDim.x) {
        if (i < nxf) {
            int f = (int)(i % (nx + 1)), iy = (int)(i / (nx + 1));
            double v;
            if (f == 0) v = s.b[CI(0, iy)];
            else if (f == nx) v = s.b[CI(nx - 1, iy)];
            else v = (s.b[CI(f, iy)] + s.b[CI(f - 1, iy)]) / 2;
            s.b_x[i] = v;
        } else {
            long long j = i - nxf;
            int ix = (int)(j % nx), f = (int)(j / nx);
            double v;
            if (f == 0) v = s.b[CI(ix, 0)];
            else if (f == ny) v = s.b[CI(ix, ny - 1)];
            else v = (s.b[CI(ix, f)] + s.b[CI(ix, f - 1)]) / 2;
            s.b_y[j] = v;
        }
    }
}
__global__ void k_gap_faces(int nx, int ny, shk_state s) { gap_faces_body(grid_blk(), nx, ny, s); }

__global__ void k_fill(size_t n, double *dst, double v, const double *base) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = base ? v + base[i] : v;
}

// ---------------------------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------------------------
static int flat_grid(Ctx *c, long long n) {
    long long b = (n + kThreads - 1) / kThreads;
    long long cap = (long long)c->num_sms * 16;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (int)b;
}

int build_mask8(Ctx *c) {
    const int n = c->nx * c->ny;
    k_mask8<<<flat_grid(c, n), kThreads, 0, c->stream>>>(n, c->st.mask, c->mask8);
    c->launches++;
    return check_launch(c, "k_mask8");
}

// One resident wave of the tail (kTailBlocksPerSm blocks per SM), or strips of two rows where those are fewer.
int tail_blocks(int nx, int ny, int num_sms) {
    const long long strips = (long long)((nx + kTailCols - 1) / kTailCols) * ((ny + 1) / 2);
    const long long blocks = (strips + kTailThreads / 32 - 1) / (kTailThreads / 32);
    return (int)std::max(1LL, std::min(blocks, (long long)num_sms * kTailBlocksPerSm));
}
template <bool FROM_H, bool CHECK>
static void run_tail(Ctx *c, const double *h_prev, PicDev *pic, const CgDev *after) {
    auto kernel = c->SL.kind == SHK_SLIDING_REG_COULOMB ? k_tail<FROM_H, CHECK, false> : k_tail<FROM_H, CHECK, true>;
    kernel<<<tail_blocks(c->nx, c->ny, c->num_sms), kTailThreads, 0, c->stream>>>(
        c->nx, c->ny, c->P, c->SL, c->st, c->mask8, h_prev, c->partials, c->counter, pic, after);
}

int launch_initial_conditions(Ctx *c) {
    const int nx = c->nx, ny = c->ny, n = nx * ny;
    const long long nf = (long long)(nx + 1) * ny + (long long)nx * (ny + 1);
    int rc = build_mask8(c);
    if (rc) return rc;
    k_face_masks_and_sliding<<<flat_grid(c, nf), kThreads, 0, c->stream>>>(nx, ny, c->mask8, c->st.valid_x,
                                                                            c->st.valid_y, c->st.ub_x, c->st.ub_y);
    c->launches++;
    if ((rc = check_launch(c, "k_face_masks_and_sliding"))) return rc;
    k_init_center<<<flat_grid(c, n), kThreads, 0, c->stream>>>(n, c->P, c->st, c->mask8);
    c->launches++;
    if ((rc = check_launch(c, "k_init_center"))) return rc;
    k_abs_ub<<<flat_grid(c, n), kThreads, 0, c->stream>>>(nx, ny, c->st);
    c->launches++;
    if ((rc = check_launch(c, "k_abs_ub"))) return rc;
    k_init_faces<<<flat_grid(c, nf), kThreads, 0, c->stream>>>(nx, ny, c->P, c->st);
    c->launches++;
    if ((rc = check_launch(c, "k_init_faces"))) return rc;
    run_tail<false, false>(c, nullptr, nullptr, nullptr);
    c->launches++;
    return check_launch(c, "k_tail<init>");
}

int launch_assemble(Ctx *c, int parabolic, double dt, bool copy_h_prev) {
    double *hp = copy_h_prev ? c->h_prev : nullptr;
    const long long tiles = (long long)((c->nx + kTX - 1) / kTX) * ((c->ny + kTY - 1) / kTY);
    const int grid = (int)std::max(1LL, std::min(tiles, (long long)c->num_sms * kAsmBlocksPerSm));
    if (parabolic)
        k_assemble<true><<<grid, kThreads, 0, c->stream>>>(c->nx, c->ny, c->P, c->kfs, dt, c->st, c->mask8,
                                                                      c->aP, c->aE, c->aN, c->rhs, hp);
    else
        k_assemble<false><<<grid, kThreads, 0, c->stream>>>(c->nx, c->ny, c->P, c->kfs, dt, c->st, c->mask8,
                                                                       c->aP, c->aE, c->aN, c->rhs, hp);
    c->launches++;
    return check_launch(c, "k_assemble");
}

int launch_export_mfls(Ctx *c, double *aP, double *aE, double *aW, double *aN, double *aS, double *rhs) {
    const int n = c->nx * c->ny;
    k_export_mfls<<<flat_grid(c, n), kThreads, 0, c->stream>>>(c->nx, c->ny, c->aP, c->aE, c->aN, c->rhs, aP, aE, aW,
                                                                aN, aS, rhs);
    c->launches++;
    return check_launch(c, "k_export_mfls");
}

int launch_tail(Ctx *c, bool picard_check, const CgDev *after) {
    if (picard_check) run_tail<true, true>(c, c->h_prev, &c->dev->pic, after);
    else run_tail<true, false>(c, nullptr, nullptr, after);
    c->launches++;
    return check_launch(c, "k_tail");
}

int launch_relax(Ctx *c, double alpha, const double *h_prev, const CgDev *after) {
    const int n = c->nx * c->ny;
    k_relax<<<flat_grid(c, n), kThreads, 0, c->stream>>>(n, alpha, c->st.h, h_prev, after);
    c->launches++;
    return check_launch(c, "k_relax");
}

int launch_step_b(Ctx *c, double dt) {
    const int nx = c->nx, ny = c->ny, n = nx * ny;
    const long long nf = (long long)(nx + 1) * ny + (long long)nx * (ny + 1);
    if (c->gap == SHK_GAP_IMPLICIT)
        k_gap_b<true><<<flat_grid(c, n), kThreads, 0, c->stream>>>(n, c->P, dt, c->st, c->mask8);
    else
        k_gap_b<false><<<flat_grid(c, n), kThreads, 0, c->stream>>>(n, c->P, dt, c->st, c->mask8);
    c->launches++;
    int rc = check_launch(c, "k_gap_b");
    if (rc) return rc;
    k_gap_faces<<<flat_grid(c, nf), kThreads, 0, c->stream>>>(nx, ny, c->st);
    c->launches++;
    return check_launch(c, "k_gap_faces");
}

int launch_fill(Ctx *c, double *dst, double v, size_t n) {
    k_fill<<<flat_grid(c, (long long)n), kThreads, 0, c->stream>>>(n, dst, v, nullptr);
    c->launches++;
    return check_launch(c, "k_fill");
}

int launch_fill_plus_base(Ctx *c, double *dst, double v, const double *base, size_t n) {
    k_fill<<<flat_grid(c, (long long)n), kThreads, 0, c->stream>>>(n, dst, v, base);
    c->launches++;
    return check_launch(c, "k_fill");
}

// ---------------------------------------------------------------------------------------------
// Ensemble: the same bodies over every instance in one grid (block -> instance table per family).
// Instances whose Picard loop has finished this timestep return at once.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_ens_assemble(EnsInst *E, const int *b2i) {
    __shared__ EnsInst I;
    const Blk B = ens_stage(I, E, b2i, EF_STENCIL);
    if (!I.pic_active) return;
    assemble_body<false>(B, I.nx, I.ny, I.P, I.kfs, 0.0, I.st, I.mask8, I.aP, I.aE, I.aN, I.rhs, I.h_prev);
}

__global__ void __launch_bounds__(kTailThreads, kTailBlocksPerSm) k_ens_tail(EnsInst *E, const int *b2i) {
    __shared__ EnsInst I;
    const Blk B = ens_stage(I, E, b2i, EF_TAIL);
    if (!I.pic_active) return;
    tail_body<true, true, true>(B, I.nx, I.ny, I.P, I.SL, I.st, I.mask8, I.h_prev, I.partials, I.counter, I.pic);
}

// step_b!: gap update of the cells, then the face averages (two launches: the faces read
// neighbouring cells' new b)
__global__ void __launch_bounds__(kThreads) k_ens_gap_cells(EnsInst *E, const int *b2i, const EnsCtl *ctl) {
    __shared__ EnsInst I;
    const Blk B = ens_stage(I, E, b2i, EF_FLAT);
    const double dt = ctl->dt;
    if (I.gap == SHK_GAP_IMPLICIT) gap_b_body<true>(B, I.nx * I.ny, I.P, dt, I.st);
    else gap_b_body<false>(B, I.nx * I.ny, I.P, dt, I.st);
}
__global__ void __launch_bounds__(kThreads) k_ens_gap_faces(EnsInst *E, const int *b2i) {
    __shared__ EnsInst I;
    const Blk B = ens_stage(I, E, b2i, EF_FLAT);
    gap_faces_body(B, I.nx, I.ny, I.st);
}

void ens_assemble(cudaStream_t s, EnsInst *E, const int *b2i, int nblocks) {
    k_ens_assemble<<<nblocks, kThreads, 0, s>>>(E, b2i);
}
void ens_tail(cudaStream_t s, EnsInst *E, const int *b2i, int nblocks) {
    k_ens_tail<<<nblocks, kTailThreads, 0, s>>>(E, b2i);
}
void ens_gap(cudaStream_t s, EnsInst *E, const int *b2i, int nblocks, const EnsCtl *ctl) {
    k_ens_gap_cells<<<nblocks, kThreads, 0, s>>>(E, b2i, ctl);
    k_ens_gap_faces<<<nblocks, kThreads, 0, s>>>(E, b2i);
}

} // namespace shk
