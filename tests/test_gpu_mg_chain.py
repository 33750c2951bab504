"""The V-cycle's kernels launched early (each starts while the previous one ends) against the same kernels
launched one by one (a process with CUDA_LAUNCH_BLOCKING=1, whose launches return when the kernel has ended).

The kernels and the order of every sum are the same, so the heads agree bit for bit, as a graph's nodes and as
plain launches: every read of an earlier kernel's output waits for it."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
# TMA-staged tiles and plain ones; level 0 with as many tiles as one wave of blocks holds, fewer and more; none
# to four levels above the bottom one
SIZES = [(2, 2), (33, 65), (96, 130), (128, 128), (385, 301), (512, 512), (512, 592), (608, 512), (901, 545), (1024, 1024)]


def solve(shk, nx, ny):
    import torch
    w = shk.configs.plain(nx, 97.0 * (nx - 1), ny=ny, ly=101.0 * (ny - 1), C=0.25)
    m = w.inputs["mask"]
    rng = np.random.default_rng(3)
    m[1:, :][rng.random((nx - 1, ny)) < 0.06] = 2.0
    g = shk.Grid(w.nx, w.ny, w.lx, w.ly)
    p, sl, s = shk.ModelParameters(), shk.RegularizedCoulombSlidingLaw(0.25), shk.State(g)
    shk.set_initial_conditions(s, g, p, sl, **w.inputs)
    gen = torch.Generator("cuda").manual_seed(5)
    s.h += torch.randn((ny, nx), generator=gen, device="cuda", dtype=torch.float64).t()
    ls = shk.CGIterativeSolver(g, shk.MatrixFreeLinearSystem, multigrid=True, stop_rule="relres", atol=0.0, rtol=0.0,
                               itmax=5)
    shk.solve_elliptic_linear_system(ls, s, g, p, shk.Arithmetic(), sl)
    return s.h.cpu().numpy()


@pytest.fixture(scope="module")
def one_by_one(cuda, tmp_path_factory):
    out = tmp_path_factory.mktemp("chain") / "h.npz"
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1", SHK_MG_RESIDENT="0", SHK_CG_GRAPHS="0")
    subprocess.run([sys.executable, __file__, str(out)], check=True, env=env, cwd=ROOT, timeout=300)
    return np.load(out)


@pytest.mark.parametrize("nx,ny", SIZES)
def test_chained_launches(shk, one_by_one, monkeypatch, nx, ny):
    monkeypatch.setenv("SHK_MG_RESIDENT", "0")
    assert np.array_equal(solve(shk, nx, ny), one_by_one[f"{nx}x{ny}"])
    monkeypatch.setenv("SHK_CG_GRAPHS", "0")
    assert np.array_equal(solve(shk, nx, ny), one_by_one[f"{nx}x{ny}"])


if __name__ == "__main__":
    sys.path.insert(0, str(ROOT))
    from __graft_entry__ import load_package
    package = load_package()
    np.savez(sys.argv[1], **{f"{nx}x{ny}": solve(package, nx, ny) for nx, ny in SIZES})
