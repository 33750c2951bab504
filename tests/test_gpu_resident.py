"""The resident solve (one persistent kernel per Jacobi or Chebyshev CG solve, shk_resident.cu) against
the general kernels (SHK_CG_RESIDENT=0) on the same systems.

The two form every element with the same operations and differ in the order of their sums only: p'Ap,
r'z, r'r and, for the Chebyshev bounds, 30 sums of the Lanczos steps.  A sum of n terms of one sign
taken in another order moves by at most n eps relative to it (2.3e-10 for 1024 x 1024 cells, and two
orders less for sums taken as trees); after a fixed small number of iterations the heads therefore agree
to 1e-10, and a converged solve to what its tolerance leaves, 1e-9, with iteration counts within 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(shk, w, monkeypatch, resident, degree, e_v=0.0, seed=5, **kw):
    monkeypatch.setenv("SHK_CG_RESIDENT", "1" if resident else "0")
    g = shk.Grid(w.nx, w.ny, w.lx, w.ly)
    p = shk.ModelParameters(e_v=e_v)
    sl = shk.RegularizedCoulombSlidingLaw(0.25)
    s = shk.State(g)
    shk.set_initial_conditions(s, g, p, sl, **w.inputs)
    import torch
    gen = torch.Generator("cuda").manual_seed(seed)
    s.h += torch.randn((w.ny, w.nx), generator=gen, device="cuda", dtype=torch.float64).t()
    ls = shk.CGIterativeSolver(g, shk.MatrixFreeLinearSystem, chebyshev_degree=degree, stop_rule="relres", atol=0.0, **kw)
    if e_v:
        st = shk.solve_parabolic_linear_system(ls, s, g, p, shk.Harmonic(), 1800.0, sl)
    else:
        st = shk.solve_elliptic_linear_system(ls, s, g, p, shk.Arithmetic(), sl)
    return s.h.cpu().numpy(), st


def workload(shk, nx, ny, blobs=False):
    w = shk.configs.plain(nx, 97.0 * (nx - 1), ny=ny, ly=101.0 * (ny - 1), C=0.25)
    if blobs:  # LAND and OTHER_BASIN cells, on strip edges too
        rng = np.random.default_rng(3)
        m = w.inputs["mask"]
        m[1:, :][rng.random((nx - 1, ny)) < 0.05] = 2.0
        m[1:, :][rng.random((nx - 1, ny)) < 0.05] = 3.0
    return w


def rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


# one block; one row group and many; odd widths; warps that end inside a row; partly filled last
# strips; every number of rows per thread; the largest grid, and one past it on each side
SIZES = [(2, 2), (3, 7), (63, 65), (64, 64), (65, 33), (129, 150), (201, 150), (256, 593), (512, 297), (513, 301),
         (640, 888), (1023, 149), (1024, 1024), (1024, 1036), (1024, 1037), (1025, 64)]


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("degree", [None, 1, 4])
def test_resident_solve_matches_general_kernels(shk, cuda, monkeypatch, nx, ny, degree):
    w = workload(shk, nx, ny, blobs=min(nx, ny) > 8)
    for e_v in (0.0, 1e-3):
        a, sa = solve(shk, w, monkeypatch, True, degree, e_v, rtol=0.0, itmax=6)
        b, sb = solve(shk, w, monkeypatch, False, degree, e_v, rtol=0.0, itmax=6)
        assert sa.status == sb.status and sa.niter == sb.niter
        assert rel(a, b) <= 1e-10
        if degree:
            assert sa.bounds_valid == sb.bounds_valid
            assert abs(sa.lambda_max - sb.lambda_max) <= 1e-9 * sb.lambda_max
            assert abs(sa.lambda_min - sb.lambda_min) <= 1e-7 * sb.lambda_max
        a, sa = solve(shk, w, monkeypatch, True, degree, e_v, rtol=1e-12)
        b, sb = solve(shk, w, monkeypatch, False, degree, e_v, rtol=1e-12)
        assert sa.status == sb.status == 0
        assert abs(sa.niter - sb.niter) <= 1 + sb.niter // 200
        assert rel(a, b) <= 1e-9


@pytest.mark.parametrize("nx,ny", [(2, 2), (2, 256), (33, 124), (37, 53), (61, 64), (64, 64), (65, 63), (97, 42),
                                   (128, 32), (127, 31)])
@pytest.mark.parametrize("rule", ["relres", "krylov"])
def test_one_block_solve_keeps_the_general_sums(shk, cuda, monkeypatch, nx, ny, rule):
    """Up to 4096 cells the resident Jacobi solve adds its sums in the order of the row-marching kernels
    (SHK_MG_TMA=0 selects them): the same head bit for bit."""
    out = []
    for tma in ("1", "0"):
        monkeypatch.setenv("SHK_MG_TMA", tma)
        w = workload(shk, nx, ny, blobs=min(nx, ny) > 8)
        g = shk.Grid(w.nx, w.ny, w.lx, w.ly)
        p, sl, s = shk.ModelParameters(), shk.RegularizedCoulombSlidingLaw(0.25), shk.State(g)
        shk.set_initial_conditions(s, g, p, sl, **w.inputs)
        kw = dict(stop_rule="relres", rtol=1e-10, atol=0.0) if rule == "relres" else {}
        ls = shk.CGIterativeSolver(g, shk.MatrixFreeLinearSystem, **kw)
        st = shk.solve_elliptic_linear_system(ls, s, g, p, shk.Arithmetic(), sl)
        out.append((s.h.cpu().numpy(), st.niter, st.status, st.rnorm, st.rnorm0))
    assert out[0][1:] == out[1][1:]
    assert np.array_equal(out[0][0], out[1][0])


def test_resident_solve_gives_up_and_recovers(shk, cuda, monkeypatch):
    """With no polls allowed a wait runs out: the solve reports it, and the next context solves."""
    w = workload(shk, 201, 150)
    monkeypatch.setenv("SHK_TEST_RESIDENT_POLLS", "0")
    with pytest.raises(shk._lib.ShaktiError, match="did not complete"):
        solve(shk, w, monkeypatch, True, None, rtol=1e-12)
    monkeypatch.delenv("SHK_TEST_RESIDENT_POLLS")
    a, sa = solve(shk, w, monkeypatch, True, None, rtol=1e-12)
    b, sb = solve(shk, w, monkeypatch, False, None, rtol=1e-12)
    assert sa.status == sb.status == 0 and rel(a, b) <= 1e-9
