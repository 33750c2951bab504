"""The basal drag on faces without sliding: the formula's value, NaN included, where the kernel leaves early."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2.5, 4.0])
@pytest.mark.parametrize("v0", [-1e-3, -1e-8, 0.0, 1e-6, np.inf, np.nan])
@pytest.mark.parametrize("still", ["ub_x", "ub_y"])
def test_drag_without_sliding_follows_the_formula(shk, orc, cuda, n, v0, still):
    """N C (|v| / (|v| + v0))^(1/n) ub / |v| with ub = 0 is NaN where the root is not finite (v0 = -|v|, v0 < -|v|),
    not 0."""
    w = shk.configs.plain(65, 97.0 * 64, ny=33, ly=101.0 * 32, C=0.25)
    w.inputs["ub_y"] = np.full((65, 34), 2e-8, order="F")
    w.inputs[still] = np.zeros_like(w.inputs[still])
    prm = dict(n=n)
    g, p = shk.Grid(w.nx, w.ny, w.lx, w.ly), shk.ModelParameters(**prm)
    sl = shk.RegularizedCoulombV0SlidingLaw(g, 0.25, v0)
    s = shk.State(g)
    shk.set_initial_conditions(s, g, p, sl, **w.inputs)
    st = orc.OracleState(w.nx, w.ny, w.lx, w.ly)
    osl = orc.SlidingSpec(kind=2, v0=v0, Cx=np.full((w.nx + 1, w.ny), 0.25, order="F"),
                          Cy=np.full((w.nx, w.ny + 1), 0.25, order="F"))
    orc.set_initial_conditions(st, prm, osl, w.inputs)
    for f in ("taub_x", "taub_y", "shear"):
        a, b = s[f].cpu().numpy(), st.fields[f]
        assert np.array_equal(np.isnan(a), np.isnan(b)), f
        # the root: CUDA's pow against the host's, a few ulp
        assert np.allclose(np.nan_to_num(a), np.nan_to_num(b), rtol=1e-13, atol=0.0), f
