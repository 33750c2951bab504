"""The resident multigrid solve (one persistent kernel per solve, shk_mg_resident.cu) against the general
kernels (SHK_MG_RESIDENT=0) on the same systems.

Both run the same V-cycle rounding for rounding and differ in the order of the dot products' sums only:
after a fixed small number of iterations the heads agree to 1e-10 (see test_gpu_resident.py), and a
converged solve to what its tolerance leaves, with iteration counts within 1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(shk, nx, ny, monkeypatch, resident, e_v=0.0, seed=5, **kw):
    monkeypatch.setenv("SHK_MG_RESIDENT", "1" if resident else "0")
    w = shk.configs.plain(nx, 97.0 * (nx - 1), ny=ny, ly=101.0 * (ny - 1), C=0.25)
    if min(nx, ny) > 8:
        rng = np.random.default_rng(3)
        m = w.inputs["mask"]
        m[1:, :][rng.random((nx - 1, ny)) < 0.06] = 2.0  # LAND and OTHER_BASIN, on strip edges too
        m[1:, :][rng.random((nx - 1, ny)) < 0.06] = 3.0
    import torch
    g = shk.Grid(w.nx, w.ny, w.lx, w.ly)
    p, sl, s = shk.ModelParameters(e_v=e_v), shk.RegularizedCoulombSlidingLaw(0.25), shk.State(g)
    shk.set_initial_conditions(s, g, p, sl, **w.inputs)
    gen = torch.Generator("cuda").manual_seed(seed)
    s.h += torch.randn((ny, nx), generator=gen, device="cuda", dtype=torch.float64).t()
    ls = shk.CGIterativeSolver(g, shk.MatrixFreeLinearSystem, multigrid=True, **kw)
    if e_v:
        st = shk.solve_parabolic_linear_system(ls, s, g, p, shk.Harmonic(), 1800.0, sl)
    else:
        st = shk.solve_elliptic_linear_system(ls, s, g, p, shk.Arithmetic(), sl)
    return s.h.cpu().numpy(), st


def rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


# one strip and many; one, two and three levels above the bottom; two and four rows per thread; odd sizes
# on every level; strips that end inside an aggregate; the widest grid and one past it
SIZES = [(2, 2), (3, 7), (17, 15), (33, 65), (64, 64), (65, 33), (96, 130), (129, 150), (200, 301), (256, 256), (257, 255),
         (301, 200), (385, 301), (511, 97), (512, 512), (512, 600), (513, 64)]


@pytest.mark.parametrize("nx,ny", SIZES)
def test_resident_multigrid_matches_general_kernels(shk, cuda, monkeypatch, nx, ny):
    for e_v in (0.0, 1e-3):
        kw = dict(stop_rule="relres", atol=0.0)
        for itmax in (1, 4):
            a, sa = solve(shk, nx, ny, monkeypatch, True, e_v, rtol=0.0, itmax=itmax, **kw)
            b, sb = solve(shk, nx, ny, monkeypatch, False, e_v, rtol=0.0, itmax=itmax, **kw)
            assert sa.status == sb.status and sa.niter == sb.niter
            assert rel(a, b) <= 1e-10
        a, sa = solve(shk, nx, ny, monkeypatch, True, e_v, rtol=1e-12, **kw)
        b, sb = solve(shk, nx, ny, monkeypatch, False, e_v, rtol=1e-12, **kw)
        assert sa.status == sb.status == 0 and abs(sa.niter - sb.niter) <= 1
        assert rel(a, b) <= 1e-9
    a, sa = solve(shk, nx, ny, monkeypatch, True)  # Krylov's rule and tolerances
    b, sb = solve(shk, nx, ny, monkeypatch, False)
    assert sa.status == sb.status and abs(sa.niter - sb.niter) <= 1


def test_resident_multigrid_gives_up_and_recovers(shk, cuda, monkeypatch):
    """With no polls allowed a wait runs out: the solve reports it, and the next context solves."""
    monkeypatch.setenv("SHK_TEST_RESIDENT_POLLS", "0")
    with pytest.raises(shk._lib.ShaktiError, match="did not complete"):
        solve(shk, 200, 150, monkeypatch, True, stop_rule="relres", rtol=1e-10, atol=0.0)
    monkeypatch.delenv("SHK_TEST_RESIDENT_POLLS")
    a, sa = solve(shk, 200, 150, monkeypatch, True, stop_rule="relres", rtol=1e-12, atol=0.0)
    b, sb = solve(shk, 200, 150, monkeypatch, False, stop_rule="relres", rtol=1e-12, atol=0.0)
    assert sa.status == sb.status == 0 and rel(a, b) <= 1e-9
