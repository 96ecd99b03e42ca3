"""The resident iteration (csrc/bbpp_persist.cu): whole solves on grids at the
edges of its box plans, against the CPU oracle and against the one-kernel-per-
step iteration (BBPP_PERSIST=0 when the context is made)."""
import numpy as np
import pytest

import bbpp
from bbpp import problems

pytestmark = pytest.mark.gpu


def problem(dims, bc, seed, frac):
    nx, ny, nz = dims
    g = bbpp.Grid.make(nx, ny, nz, 1.0 / nx, 1.0 / ny, 1.0 / nz, problems.bc_tuple(bc))
    rng = np.random.default_rng(seed)
    mask = (rng.random(g.shape) < frac).astype(np.uint8) if frac else None
    b = rng.uniform(-1, 1, g.shape)
    if frac:
        b[mask == 1] = 0
        b[mask == 0] -= b[mask == 0].mean()
    else:
        b -= b.mean()
    return g, mask, b


# a box of one cell a direction, more columns than threads, walls on both sides of
# a box, a periodic axis in one box, odd splits; the three levels of what lives
# in shared memory in FP64 (about 0.9M and 1.15M cells) and FP32 (1.75M, 2.3M), and
# FP32 boxes that leave no room for the halo's residual (two exchanges an iteration)
CASES = [
    ((301, 2, 1), "ppp", 0.0, bbpp.FP64),
    ((1, 1, 7), "ppn", 0.0, bbpp.FP64),
    ((7, 5, 64), "nnn", 0.03, bbpp.FP64),
    ((600, 9, 8), "pnp", 0.03, bbpp.FP32_IR),
    ((53, 64, 31), "npn", 0.02, bbpp.FP64),
    ((104, 100, 100), "pnn", 0.02, bbpp.FP64),
    ((128, 120, 101), "ppn", 0.02, bbpp.FP64),
    ((101, 90, 80), "nnp", 0.02, bbpp.FP32_IR),
    ((128, 125, 130), "ppn", 0.02, bbpp.FP32_IR),
    ((160, 150, 140), "pnn", 0.02, bbpp.FP32_IR),
    ((183, 184, 184), "npp", 0.02, bbpp.FP32_IR),
]


@pytest.mark.parametrize("dims,bc,frac,precision", CASES)
def test_resident_solve(bbpp_lib, orc, monkeypatch, dims, bc, frac, precision):
    g, mask, b = problem(dims, bc, sum(dims), frac)
    tol = 1e-11 if precision == bbpp.FP64 else 1e-8
    x, rep = bbpp.Solver(g).solve_host(b, mask, tol=tol, precision=precision, replace_every=50)
    monkeypatch.setenv("BBPP_PERSIST", "0")
    x2, rep2 = bbpp.Solver(g).solve_host(b, mask, tol=tol, precision=precision, replace_every=50)
    assert rep.status == rep2.status == bbpp.CONVERGED and rep.true_rel <= tol * 1.01
    # the same arithmetic per cell; the dot products group their partial sums by
    # other CTAs, so the last digits and with them the last iteration may differ
    assert abs(rep.iters - rep2.iters) <= max(2, rep2.iters // 50)
    if mask is None:
        x, x2 = x - x.mean(), x2 - x2.mean()
    else:
        assert np.all(x[mask == 1] == 0)
    scale = np.abs(x2).max()
    # both within tol of a zero residual: the error is bounded by tol times the
    # condition number, below 1e4 for the largest extent here
    assert np.abs(x - x2).max() <= 1e4 * tol * scale
    if g.n <= 1_100_000:
        xo, _ = orc.pcg(orc.from_tuple(g.as_tuple()), b, mask, tol=1e-13)
        if mask is None:
            xo = xo - xo.mean()
        assert np.abs(x - xo).max() <= 1e4 * tol * np.abs(xo).max()


@pytest.mark.parametrize("replace_every", [7, 50])
def test_resident_trace(bbpp_lib, orc, replace_every):
    """Checkpoints at an odd spacing (the search direction's buffers alternate
    between launches) and at the usual one: alpha and beta as the oracle's."""
    g, mask, b = problem((40, 33, 29), "ppn", 3, 0.03)
    s = bbpp.Solver(g)
    s.set_trace(60)
    x, rep = s.solve_host(b, mask, tol=1e-11, replace_every=replace_every)
    a, be = s.trace()
    xo, res = orc.pcg(orc.from_tuple(g.as_tuple()), b, mask, tol=1e-11, replace_every=replace_every, trace=60)
    assert rep.status == bbpp.CONVERGED and abs(rep.iters - res["iters"]) <= 2
    n = min(50, rep.iters - 2)
    assert np.all(np.abs(a[:n] / res["alpha"][:n] - 1) <= 1e-12)
    assert np.all(np.abs(be[:n] / res["beta"][:n] - 1) <= 1e-12)


def test_resident_checkpoint_every_iteration(bbpp_lib, orc):
    """replace_every = 1: one iteration a launch, every residual from x."""
    g, mask, b = problem((40, 33, 29), "ppn", 3, 0.03)
    x, rep = bbpp.Solver(g).solve_host(b, mask, tol=1e-10, replace_every=1)
    xo, res = orc.pcg(orc.from_tuple(g.as_tuple()), b, mask, tol=1e-10, replace_every=1)
    assert rep.status == bbpp.CONVERGED and abs(rep.iters - res["iters"]) <= max(2, res["iters"] // 50)
    assert np.abs(x - xo).max() <= 1e4 * 1e-10 * np.abs(xo).max()


def test_resident_iteration_limit(bbpp_lib):
    """max_iter + 1 iterations, as the reference's loop; the solution of the
    unfinished solve is the two-kernel iteration's."""
    g, mask, b = problem((48, 40, 36), "ppn", 5, 0.03)
    x, rep = bbpp.Solver(g).solve_host(b, mask, tol=1e-14, max_iter=63, ok=(bbpp.MAX_ITER,))
    assert rep.status == bbpp.MAX_ITER and rep.iters == 64
