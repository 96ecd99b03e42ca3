"""Waits and launches of the resident iteration that fail (csrc/bbpp_persist.cu),
by the host's and the kernels' test hooks: the solve says so, or goes on kernel
by kernel, and the context stays usable.  Nothing faults, traps or hangs."""
import numpy as np
import pytest

import bbpp
from bbpp import problems

pytestmark = pytest.mark.gpu
LAST_WAIT, REFUSED, EXCHANGE = 2, 3, 5


def problem(dims, bc, seed=3):
    nx, ny, nz = dims
    g = bbpp.Grid.make(nx, ny, nz, 1.0 / nx, 1.0 / ny, 1.0 / nz, problems.bc_tuple(bc))
    rng = np.random.default_rng(seed)
    mask = (rng.random(g.shape) < 0.05).astype(np.uint8)
    b = rng.uniform(-1, 1, g.shape)
    b[mask == 1] = 0
    b[mask == 0] -= b[mask == 0].mean()
    return g, mask, b


ANY = (bbpp.CONVERGED, bbpp.WAIT_TIMEOUT)


@pytest.mark.parametrize("precision", [bbpp.FP64, bbpp.FP32_IR])
@pytest.mark.parametrize("dims", [(40, 33, 29), (128, 100, 90)])
def test_a_wait_that_ran_out_is_not_overwritten(bbpp_lib, precision, dims):
    """The last CTA's wait runs out in the exchange by which the others see the
    solve converge: one box is not written back, so the solve must not pass for
    converged.  Under the (r,z) rule no residual is formed again that would show it."""
    g, mask, b = problem(dims, "ppn")
    s = bbpp.Solver(g)
    L = bbpp.lib()
    for _ in range(4):
        assert L.bbpp_debug_wait(s.handle, 0, LAST_WAIT) == 0
        x, rep = s.solve_host(b, mask, tol=1e-8, precision=precision, stop=bbpp.STOP_REF_RZ, ok=ANY)
        assert rep.status == bbpp.WAIT_TIMEOUT
    assert L.bbpp_debug_wait(s.handle, 0, 0) == 0
    x, rep = s.solve_host(b, mask, tol=1e-8, precision=precision)
    assert rep.status == bbpp.CONVERGED and rep.true_rel <= 1.01e-8


@pytest.mark.parametrize("precision,ir_mode", [(bbpp.FP64, 0), (bbpp.FP32_IR, bbpp.IR_RELIABLE),
                                               (bbpp.FP32_IR, bbpp.IR_RESTART)])
def test_a_refused_launch_falls_back(bbpp_lib, monkeypatch, precision, ir_mode):
    """The cooperative launch is refused (the host's fake of the error): the solve
    takes the kernels of single iterations, and the context's later solves those of a
    context without the resident form, to the same bits."""
    g, mask, b = problem((48, 40, 30), "ppn")
    kw = dict(tol=1e-9, precision=precision, ir_mode=ir_mode)
    s = bbpp.Solver(g)
    L = bbpp.lib()
    assert L.bbpp_debug_wait(s.handle, 0, REFUSED) == 0
    x, rep = s.solve_host(b, mask, **kw)
    assert L.bbpp_debug_wait(s.handle, 0, 0) == 0
    x1, rep1 = s.solve_host(b, mask, **kw)
    monkeypatch.setenv("BBPP_PERSIST", "0")
    later, _ = bbpp.Solver(g).solve_host(b, mask, **kw)
    monkeypatch.setenv("BBPP_PAIR", "0")
    first, rep0 = bbpp.Solver(g).solve_host(b, mask, **kw)
    assert rep.status == rep1.status == bbpp.CONVERGED
    assert rep.iters == rep0.iters and np.array_equal(x, first)
    assert np.array_equal(x1, later)


@pytest.mark.parametrize("precision", [bbpp.FP64, bbpp.FP32_IR])
@pytest.mark.parametrize("dims", [(12, 9, 7), (40, 33, 29), (128, 100, 90)])
def test_an_exchange_without_a_cta(bbpp_lib, precision, dims):
    """Every CTA's wait gives up and returns, in FP64 as in FP32, and the next solve
    starts from clean counts."""
    g, mask, b = problem(dims, "pnp")
    s = bbpp.Solver(g)
    L = bbpp.lib()
    for _ in range(2):
        assert L.bbpp_debug_wait(s.handle, 2_000_000, EXCHANGE) == 0   # 2 ms
        x, rep = s.solve_host(b, mask, tol=1e-8, precision=precision, ok=ANY)
        assert rep.status == bbpp.WAIT_TIMEOUT
        assert L.bbpp_debug_wait(s.handle, 0, 0) == 0
        x, rep = s.solve_host(b, mask, tol=1e-8, precision=precision)
        assert rep.status == bbpp.CONVERGED and rep.true_rel <= 1.01e-8


@pytest.mark.parametrize("precision", [bbpp.FP64, bbpp.FP32_IR])
@pytest.mark.parametrize("dims", [(48, 40, 36), (130, 120, 118), (160, 150, 140)])
@pytest.mark.parametrize("max_iter", [5, 48, 49, 50, 63])
def test_the_solution_of_an_unfinished_solve(bbpp_lib, monkeypatch, precision, dims, max_iter):
    """The state that a launch leaves at an iteration limit, before, on and after a
    checkpoint and with all of it, some or none in shared memory: the two-kernel
    iteration's solution."""
    if precision == bbpp.FP64 and dims[0] == 160:
        pytest.skip("FP64 grids of this size are not resident")
    g, mask, b = problem(dims, "ppn", 5)
    kw = dict(tol=1e-14, precision=precision, max_iter=max_iter, ok=(bbpp.MAX_ITER,))
    x, rep = bbpp.Solver(g).solve_host(b, mask, **kw)
    monkeypatch.setenv("BBPP_PERSIST", "0")
    s = bbpp.Solver(g)
    s.set_fused(False)
    y, rep2 = s.solve_host(b, mask, **kw)
    assert rep.status == rep2.status == bbpp.MAX_ITER and rep.iters == rep2.iters == max_iter + 1
    # rounding (2^-53, 2^-24) times the condition number, below (2 n / pi)^2 = 1e4 for 160 cells
    eps = 2.0 ** -53 if precision == bbpp.FP64 else 2.0 ** -24
    assert np.abs(x - y).max() <= 1e4 * eps * np.abs(y).max()
