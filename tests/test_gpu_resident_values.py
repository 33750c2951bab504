"""Values out of the ordinary in the resident solves (shk_resident.cu): what the general kernels make of them."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one block, one, two and four rows per thread with stored reciprocals, and seven without
@pytest.mark.parametrize("nx,ny", [(37, 53), (201, 150), (512, 297), (640, 300), (1024, 300)])
@pytest.mark.parametrize("degree", [None, 1, 4])
@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("rule", ["relres", "krylov"])
def test_a_right_hand_side_that_is_not_finite(shk, cuda, monkeypatch, nx, ny, degree, value, rule):
    """Status, iterations, norms and head are those of the general kernels: an infinite residual stays
    infinite under the preconditioner (a quotient by a stored reciprocal included)."""
    out = []
    for resident in ("1", "0"):
        monkeypatch.setenv("SHK_CG_RESIDENT", resident)
        w = shk.configs.plain(nx, 97.0 * (nx - 1), ny=ny, ly=101.0 * (ny - 1), C=0.25)
        g, p, sl = shk.Grid(nx, ny, w.lx, w.ly), shk.ModelParameters(), shk.RegularizedCoulombSlidingLaw(0.25)
        s = shk.State(g)
        shk.set_initial_conditions(s, g, p, sl, **w.inputs)
        s.ieb[nx // 3, ny // 2] = value
        kw = dict(stop_rule="relres", rtol=1e-8, atol=0.0) if rule == "relres" else {}
        ls = shk.CGIterativeSolver(g, shk.MatrixFreeLinearSystem, chebyshev_degree=degree, **kw)
        st = shk.solve_elliptic_linear_system(ls, s, g, p, shk.Arithmetic(), sl)
        out.append((st.status, st.niter, str(st.rnorm0), str(st.rnorm), np.nan_to_num(s.h.cpu().numpy(), nan=-7e77)))
    assert out[0][:4] == out[1][:4]
    assert np.array_equal(out[0][4], out[1][4])
