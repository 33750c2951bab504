"""bench.py's count of the bytes that the default multigrid kernels move (the numerator of its fractions): z as the
Float32 value that is stored, and the bottom kernel's levels by its own rule."""
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


def test_moved_iteration_bytes(monkeypatch):
    monkeypatch.delenv("SHK_MG_FUSED", raising=False)
    n0 = 4096 * 4096
    # matvec 52 B (z 4, p_old, aP, aE, aN 32 in, p_new, Ap 16 out), level 0 62 + 34 B, levels 1-5 on tiles, levels
    # 6-12 (64 x 64 and below) in the bottom kernel
    coarse = sum((4096 >> l) ** 2 for l in range(1, 6))
    bottom = 25 * 64 * 64 + 17 * sum((64 >> k) ** 2 for k in range(1, 7))
    expect = (52 + 62 + 34) * n0 + 56 * coarse + bottom
    assert bench.iteration_bytes("multigrid", 4096, 4096, moved=True) == expect
    assert abs(expect / n0 - 166.65) < 0.01
    assert bench.iteration_bytes("plain", 4096, 4096, moved=True) == 112 * n0


@pytest.mark.parametrize("kind", ["0", "2"])
def test_forms_with_float64_z(monkeypatch, kind):
    monkeypatch.setenv("SHK_MG_FUSED", kind)
    assert bench.iteration_bytes("multigrid", 1024, 1024, moved=True) == bench.iteration_bytes("multigrid", 1024, 1024)


@pytest.mark.parametrize("n,level", [(4096, 6), (1024, 4), (385, 3), (64, 1), (129, 2)])
def test_bottom_level(n, level):
    """The finest bottom level of square grids: 64 x 64 and below (129 -> 65 -> 33)."""
    assert bench.bottom_level(bench.mg_dims(n, n)) == level


def test_step_fraction_counts_the_same_bytes(monkeypatch):
    monkeypatch.delenv("SHK_MG_FUSED", raising=False)

    class W:
        nx = ny = 4096

    counts = {"picard_iters": 46, "cg_iters": 160, "steps": 16}
    b = bench.step_bytes("multigrid", 4096, 4096, counts, moved=True)
    r = bench.step_roofline("multigrid", W, counts, 14.56, {"hbm_gbs": 6545.0}, moved=True)
    assert abs(r["achieved"] - b / 14.56e-3 / 1e9) < 0.1 and "166.7 B/cell" in r["accounting"]
    assert bench.step_bytes("multigrid", 4096, 4096, counts) - b == 10 * (
        bench.iteration_bytes("multigrid", 4096, 4096) - bench.iteration_bytes("multigrid", 4096, 4096, moved=True))
