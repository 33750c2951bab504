"""The register-resident bottom kernel of the V-cycle (k_mg_bottom) against the general one-block form
(SHK_MG_BOTTOM=0): both spell out the same roundings, so a solve gives the same head bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def solve(shk, nx, ny, monkeypatch, bottom, law):
    monkeypatch.setenv("SHK_MG_BOTTOM", bottom)
    w = shk.configs.plain(nx, 97.0 * (nx - 1), ny=ny, ly=101.0 * (ny - 1), C=0.25)
    m = w.inputs["mask"]
    rng = np.random.default_rng(3)
    m[1:, :][rng.random((nx - 1, ny)) < 0.08] = 2.0  # LAND and OTHER_BASIN: inactive cells on every level
    m[1:, :][rng.random((nx - 1, ny)) < 0.08] = 3.0
    g = shk.Grid(w.nx, w.ny, w.lx, w.ly)
    p, sl, s = shk.ModelParameters(), shk.RegularizedCoulombSlidingLaw(0.25), shk.State(g)
    shk.set_initial_conditions(s, g, p, sl, **w.inputs)
    ls = shk.CGIterativeSolver(g, shk.MatrixFreeLinearSystem, multigrid=True, stop_rule="relres", rtol=1e-9, atol=0.0)
    st = shk.solve_elliptic_linear_system(ls, s, g, p, law, sl)
    return s.h.cpu().numpy(), st


# bottoms with 0, 1, 2 and 3 column levels above the one-warp levels; full and partly filled columns;
# odd sizes on every level; long thin grids, whose levels shrink along one side only
@pytest.mark.parametrize("nx,ny", [(2, 2), (5, 7), (16, 16), (17, 15), (31, 33), (64, 64), (65, 127), (128, 128),
                                   (126, 130), (385, 301), (513, 250), (2, 700), (900, 3), (1040, 24), (520, 516),
                                   (8, 1500), (1026, 16), (4098, 5)])
def test_bottom_kernel_matches_general_form(shk, cuda, monkeypatch, nx, ny):
    a, sa = solve(shk, nx, ny, monkeypatch, "1", shk.Arithmetic())
    b, sb = solve(shk, nx, ny, monkeypatch, "0", shk.Arithmetic())
    assert sa.status == sb.status == 0 and sa.niter == sb.niter
    assert np.array_equal(a, b)
