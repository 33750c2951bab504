"""Timesteps whose solves run resident against the same by the general kernels, where a loose stopping rule and a
large sliding coefficient let the Picard loop amplify a sum taken in another order (the Jacobi solves of at
most 4096 cells keep the general order, the Chebyshev ones do not).

Bound: both Picard loops end when max|dh| <= 1e-6 max|h|, so each is within 1e-6 / (1 - q) of the loop's fixed
point, q < 1 its contraction; with q <= 0.6 over four steps that is 1e-5 of max|h| at most."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(64, 64), (37, 53), (90, 70)])
@pytest.mark.parametrize("degree", [4, 1])
def test_chebyshev_timesteps(shk, cuda, monkeypatch, nx, ny, degree):
    out = []
    for resident in ("1", "0"):
        monkeypatch.setenv("SHK_CG_RESIDENT", resident)
        w = shk.configs.plain(nx, 10e3, ny=ny, ly=10e3, C=1e4)
        g, p, sl = shk.Grid(w.nx, w.ny, w.lx, w.ly), shk.ModelParameters(), shk.RegularizedCoulombSlidingLaw(1e4)
        s = shk.State(g)
        shk.set_initial_conditions(s, g, p, sl, **w.inputs)
        ls = shk.CGIterativeSolver(g, shk.MatrixFreeLinearSystem, chebyshev_degree=degree)
        ps = shk.PicardSolver(500, 1e-6, ls, g)
        sim = shk.Simulation(g, s, 4, 1800.0, p, "implicit", [], shk.ConstantMeltInput(), sl, ps=ps)
        shk.run(sim)
        assert all(x["converged"] for x in sim.step_stats)
        out.append(s.h.cpu().numpy())
    assert np.max(np.abs(out[0] - out[1])) <= 1e-5 * np.max(np.abs(out[1]))
