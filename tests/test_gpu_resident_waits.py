"""The bounded waits of the resident solves (shk_resident.cuh), cut short."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HOOKS = ("POLLS", "BLOCK", "ITER", "ABSENT")


class Problem:
    """A perturbed state and its solver; `hooks` are the test switches a context reads when it is created."""

    def __init__(self, shk, monkeypatch, nx, ny, precond, resident=True, **hooks):
        for k in HOOKS:
            monkeypatch.delenv("SHK_TEST_RESIDENT_" + k, raising=False)
        for k, v in hooks.items():
            monkeypatch.setenv("SHK_TEST_RESIDENT_" + k, str(v))
        for k in ("CG", "MG"):
            monkeypatch.setenv(f"SHK_{k}_RESIDENT", "1" if resident else "0")
        import torch
        w = shk.configs.plain(nx, 97.0 * (nx - 1), ny=ny, ly=101.0 * (ny - 1), C=0.25)
        self.shk, self.g, self.p, self.sl = shk, shk.Grid(nx, ny, w.lx, w.ly), shk.ModelParameters(), \
            shk.RegularizedCoulombSlidingLaw(0.25)
        self.s = shk.State(self.g)
        shk.set_initial_conditions(self.s, self.g, self.p, self.sl, **w.inputs)
        gen = torch.Generator("cuda").manual_seed(5)
        self.s.h += torch.randn((ny, nx), generator=gen, device="cuda", dtype=torch.float64).t()
        self.h0 = self.s.h.clone()
        self.kw = dict(chebyshev_degree=4 if precond == "chebyshev" else None, multigrid=precond == "multigrid")

    def solver(self, **kw):
        return self.shk.CGIterativeSolver(self.g, self.shk.MatrixFreeLinearSystem, stop_rule="relres", atol=0.0,
                                          **self.kw, **kw)

    def solve(self, **kw):
        """(head, stats); without stats after an error; from the same head every time."""
        self.s.h.copy_(self.h0)
        try:
            st = self.shk.solve_elliptic_linear_system(self.solver(**kw), self.s, self.g, self.p,
                                                       self.shk.Arithmetic(), self.sl)
        except self.shk._lib.ShaktiError as e:
            assert "did not complete" in str(e)
            return self.s.h.cpu().numpy(), None
        return self.s.h.cpu().numpy(), st


FORMS = [(201, 150, "jacobi"), (640, 300, "jacobi"), (64, 64, "chebyshev"), (513, 301, "chebyshev"),
         (200, 150, "multigrid"), (385, 301, "multigrid")]


@pytest.mark.parametrize("nx,ny,precond", FORMS)
def test_a_block_whose_wait_ran_out_leaves_as_a_whole(shk, cuda, monkeypatch, nx, ny, precond):
    """Whichever warps of a block see the wait run out first: every call returns, and a context with its
    waits whole solves as before."""
    kw = dict(rtol=0.0, itmax=6)
    want, _ = Problem(shk, monkeypatch, nx, ny, precond).solve(**kw)
    for polls in (0, 1, 2, 3, 5, 8):
        q = Problem(shk, monkeypatch, nx, ny, precond, POLLS=polls)
        for _ in range(5):
            q.solve(**kw)
    h, _ = Problem(shk, monkeypatch, nx, ny, precond).solve(**kw)
    assert np.array_equal(h, want)


@pytest.mark.parametrize("block", [0, 1, 3])
@pytest.mark.parametrize("nx,ny,precond", [(64, 64, "chebyshev"), (200, 150, "multigrid")])
def test_a_sum_completes_from_whole_partials_only(shk, cuda, monkeypatch, nx, ny, precond, block):
    """One block's waits end inside the preconditioner of the last iteration, whose result enters the last
    sums: the solve ends in an error, or with every block's rows in its norms."""
    kw = dict(rtol=0.0, itmax=3)
    _, ref = Problem(shk, monkeypatch, nx, ny, precond).solve(**kw)
    q = Problem(shk, monkeypatch, nx, ny, precond, POLLS=0, BLOCK=block, ITER=3)
    for _ in range(2):
        _, st = q.solve(**kw)
        if st is not None:
            assert (st.niter, st.status, st.rnorm, st.rnorm0) == (ref.niter, ref.status, ref.rnorm, ref.rnorm0)


@pytest.mark.parametrize("block", [0, 1, 2, -1])
@pytest.mark.parametrize("nx,ny,precond", FORMS)
def test_a_solve_has_one_outcome(shk, cuda, monkeypatch, nx, ny, precond, block):
    """One block's wait (-1: every block's) for the last sum runs out while the others have it: the solve
    is reported and whole, or an error and the head untouched."""
    kw = dict(rtol=0.0, itmax=3)
    want, ref = Problem(shk, monkeypatch, nx, ny, precond).solve(**kw)
    q = Problem(shk, monkeypatch, nx, ny, precond, POLLS=0, BLOCK=block, ITER=3)
    for _ in range(4):
        h, st = q.solve(**kw)
        if st is None:
            assert np.array_equal(h, q.h0.cpu().numpy())
        else:
            assert np.array_equal(h, want) and (st.niter, st.rnorm) == (ref.niter, ref.rnorm)


@pytest.mark.parametrize("alpha", [None, 0.7])
@pytest.mark.parametrize("nx,ny,precond", [(201, 150, "jacobi"), (64, 64, "chebyshev"), (200, 150, "multigrid")])
def test_a_failed_solve_leaves_the_fields(shk, cuda, monkeypatch, nx, ny, precond, alpha):
    """The Picard loop queues head relaxation and the field update behind a solve before it knows the
    outcome: after a solve that failed neither has written anything."""
    q = Problem(shk, monkeypatch, nx, ny, precond, POLLS=0)
    before = {f: q.s[f].clone() for f in shk._lib.STATE_FIELDS}
    ps = shk.PicardSolver(5, 1e-6, q.solver(rtol=1e-10), q.g, alpha=alpha)
    with pytest.raises(shk._lib.ShaktiError, match="did not complete"):
        shk.Picard_loop(ps, q.s, q.g, q.p, None, shk.Arithmetic(), q.sl)
    for f, t in before.items():
        assert cuda.equal(q.s[f], t), f


@pytest.mark.parametrize("block", [0, 2])
@pytest.mark.parametrize("nx,ny,precond", FORMS)
def test_a_solve_that_cannot_start_runs_by_the_general_kernels(shk, cuda, monkeypatch, nx, ny, precond, block):
    """A block of the launch that does not start (another stream's kernel holds its SM): the same head, bit
    for bit, as by the general kernels, and no error; in the Picard loop too, where the warm start and
    the relaxation come after it."""
    out = []
    for resident, hooks in ((False, {}), (True, dict(ABSENT=block))):
        q = Problem(shk, monkeypatch, nx, ny, precond, resident=resident, **hooks)
        h, st = q.solve(rtol=1e-10)
        ps = shk.PicardSolver(2, 1e-30, q.solver(rtol=1e-8), q.g, alpha=0.7)
        q.s.h.copy_(q.h0)
        shk.Picard_loop(ps, q.s, q.g, q.p, None, shk.Arithmetic(), q.sl)
        out.append((h, st.niter, st.status, st.rnorm, ps.cg_iters_total, {f: q.s[f].clone() for f in shk._lib.STATE_FIELDS}))
    a, b = out
    assert np.array_equal(a[0], b[0]) and a[1:5] == b[1:5] and a[2] == 0
    for f, t in a[5].items():
        assert cuda.equal(b[5][f], t), f


@pytest.mark.parametrize("nx,ny,precond", [(201, 150, "jacobi"), (64, 64, "chebyshev"), (200, 150, "multigrid")])
def test_the_wait_for_a_start_is_paid_once_in_a_while(shk, cuda, monkeypatch, nx, ny, precond):
    """After a solve that could not start, the context's next 32 do not try (each try waits about 40 ms); the one
    after them does: it launches one kernel more."""
    q = Problem(shk, monkeypatch, nx, ny, precond, ABSENT=0)
    ls, counts = q.solver(rtol=0.0, itmax=3), []
    for _ in range(36):
        n = ls.ctx.launches()
        q.s.h.copy_(q.h0)
        shk.solve_elliptic_linear_system(ls, q.s, q.g, q.p, shk.Arithmetic(), q.sl)
        counts.append(ls.ctx.launches() - n)
    general = counts[1]
    assert [k for k, c in enumerate(counts) if c > general] == [0, 33]
    assert all(c == general for k, c in enumerate(counts) if k not in (0, 33))


def test_two_solves_at_once(shk, cuda, monkeypatch):
    """Two host threads on two streams: each gets its own solution, whether the two launches follow one
    another or one gives way to the general kernels (to 1e-9, as between the two forms)."""
    from concurrent.futures import ThreadPoolExecutor
    forms = [(640, 300, "jacobi"), (385, 301, "multigrid")]
    want = [Problem(shk, monkeypatch, *f).solve(rtol=1e-11)[0] for f in forms]
    qs = []
    for f in forms:
        stream = cuda.cuda.Stream()
        with cuda.cuda.stream(stream):
            qs.append((stream, Problem(shk, monkeypatch, *f)))
    cuda.cuda.synchronize()

    def work(k):
        stream, q = qs[k]
        with cuda.cuda.stream(stream):
            return [q.solve(rtol=1e-11) for _ in range(20)]
    with ThreadPoolExecutor(2) as ex:
        runs = list(ex.map(work, range(2)))
    for k, run in enumerate(runs):
        for h, st in run:
            assert st is not None and st.status == 0
            assert np.max(np.abs(h - want[k])) <= 1e-9 * np.max(np.abs(want[k]))


@pytest.mark.parametrize("nx,ny,precond", [(640, 300, "jacobi"), (513, 301, "chebyshev"), (385, 301, "multigrid")])
def test_a_part_of_the_device(shk, cuda, monkeypatch, nx, ny, precond):
    """A stream on 16 SMs, too few for the launch's blocks: the general kernels' head, bit for bit."""
    kw = dict(rtol=0.0, itmax=20)
    want, ref = Problem(shk, monkeypatch, nx, ny, precond, resident=False).solve(**kw)
    part = cuda.cuda.GreenContext.create(16, 0)
    stream = part.Stream()
    with cuda.cuda.stream(stream):
        h, st = Problem(shk, monkeypatch, nx, ny, precond).solve(**kw)
    gc.collect()  # the solver contexts synchronise their stream when they go: before it does
    cuda.cuda.synchronize()
    del stream, part
    assert (st.niter, st.status) == (ref.niter, ref.status) and np.array_equal(h, want)
