"""Pairs of FP32 iterations (csrc/bbpp_pair.cu), whole mixed-precision solves on
grids at the edges of its slabs and rings, against the CPU oracle and against one
iteration at a time.  BBPP_PERSIST=0 keeps small grids off the resident
iteration, BBPP_PAIR=0 off the pairs (read when the context is made)."""
import numpy as np
import pytest

import bbpp
from bbpp import problems

pytestmark = pytest.mark.gpu


def problem(dims, bc, seed, frac, iso):
    nx, ny, nz = dims
    d = (1.0 / max(dims),) * 3 if iso else (1.0 / nx, 1.0 / ny, 1.0 / nz)
    g = bbpp.Grid.make(nx, ny, nz, *d, problems.bc_tuple(bc))
    rng = np.random.default_rng(seed)
    mask = (rng.random(g.shape) < frac).astype(np.uint8) if frac else None
    b = rng.uniform(-1, 1, g.shape)
    if frac:
        b[mask == 1] = 0
        b[mask == 0] -= b[mask == 0].mean()
    else:
        b -= b.mean()
    return g, mask, b


# rows of one, three, 25 and 50 float4 (warps across rows), of a warp's multiples and
# of 1024 cells; ny of a wrapped slab, less than a slab, odd, a slab and a row; nz of
# one to five planes (rings shorter than the march) and of several chunks; walls and
# periodic axes; isotropic and not; with and without solid cells
CASES = [
    ((4, 40, 37), "ppp", 0.02, True),
    ((12, 3, 50), "ppn", 0.02, False),
    ((100, 31, 1), "pnp", 0.02, True),
    ((200, 15, 2), "nnn", 0.02, False),
    ((64, 63, 3), "ppp", 0.0, True),
    ((96, 45, 64), "npn", 0.03, True),
    ((256, 15, 40), "ppn", 0.03, True),
    ((256, 29, 5), "pnp", 0.0, False),
    ((512, 13, 33), "ppn", 0.03, True),
    ((1024, 5, 20), "ppn", 0.02, True),
    ((128, 61, 70), "ppp", 0.03, False),
]


@pytest.mark.parametrize("dims,bc,frac,iso", CASES)
def test_pair_solve(bbpp_lib, orc, monkeypatch, dims, bc, frac, iso):
    g, mask, b = problem(dims, bc, sum(dims), frac, iso)
    tol = 1e-8
    monkeypatch.setenv("BBPP_PERSIST", "0")
    x, rep = bbpp.Solver(g).solve_host(b, mask, tol=tol, precision=bbpp.FP32_IR)
    monkeypatch.setenv("BBPP_PAIR", "0")
    x2, rep2 = bbpp.Solver(g).solve_host(b, mask, tol=tol, precision=bbpp.FP32_IR)
    assert rep.status == rep2.status == bbpp.CONVERGED and rep.true_rel <= tol * 1.01
    assert abs(rep.iters - rep2.iters) <= max(4, rep2.iters // 10)
    xo, _ = orc.pcg(orc.from_tuple(g.as_tuple()), b, mask, tol=1e-13)
    if mask is None:
        x, xo = x - x.mean(), xo - xo.mean()
    else:
        assert np.all(x[mask == 1] == 0)
    # both within tol of a zero residual: the error is bounded by tol times the
    # condition number, below (2 n / pi)^2 for n cells along the longest axis
    assert np.abs(x - xo).max() <= (2 * max(dims) / np.pi) ** 2 * tol * np.abs(xo).max()


@pytest.mark.parametrize("replace_every,max_iter", [(1, 20000), (7, 20000), (50, 40), (50, 41)])
def test_pair_checkpoints_and_limit(bbpp_lib, monkeypatch, replace_every, max_iter):
    """Odd checkpoint spacings and iteration limits end on a single step."""
    g, mask, b = problem((64, 45, 30), "ppn", 9, 0.03, True)
    monkeypatch.setenv("BBPP_PERSIST", "0")
    x, rep = bbpp.Solver(g).solve_host(b, mask, tol=1e-8, precision=bbpp.FP32_IR, replace_every=replace_every,
                                       max_iter=max_iter, ok=(bbpp.CONVERGED, bbpp.MAX_ITER))
    if max_iter < 100:
        assert rep.status == bbpp.MAX_ITER and rep.iters == max_iter + 1
    else:
        assert rep.status == bbpp.CONVERGED and rep.true_rel <= 1e-8 * 1.01


def test_pair_reports_wait_timeout_and_recovers(bbpp_lib, monkeypatch):
    """A step whose copies are never issued (the test hook): its waits run out,
    the solve reports it, and the next one converges."""
    g, mask, b = problem((64, 45, 30), "ppn", 11, 0.03, True)
    monkeypatch.setenv("BBPP_PERSIST", "0")
    s = bbpp.Solver(g)
    L = bbpp.lib()
    assert L.bbpp_debug_wait(s.handle, 2_000_000, 1) == 0
    x, rep = s.solve_host(b, mask, tol=1e-8, precision=bbpp.FP32_IR, ok=(bbpp.WAIT_TIMEOUT,))
    assert rep.status == bbpp.WAIT_TIMEOUT
    assert L.bbpp_debug_wait(s.handle, 0, 0) == 0
    x, rep = s.solve_host(b, mask, tol=1e-8, precision=bbpp.FP32_IR)
    assert rep.status == bbpp.CONVERGED and rep.true_rel <= 1e-8 * 1.01


@pytest.mark.parametrize("dims,bc", [((40, 33, 37), "nnn"), ((24, 31, 40), "ppn"), ((33, 33, 33), "nnn"),
                                     ((160, 160, 160), "ppp")])
@pytest.mark.parametrize("resident", ["0", "1"])
def test_lost_residual(bbpp_lib, monkeypatch, dims, bc, resident):
    """So many solid cells that FP32 gains more than seven digits between two
    replacements: the replaced residual is far from the recursion's, and the
    iterations restart from it.  A restart reduces the residual by the six digits
    that FP32 holds at least, so 1e-8 takes two of them: three times the FP64
    iterations, and what is left to the next checkpoint each time."""
    monkeypatch.setenv("BBPP_PERSIST", resident)
    g, mask, b = problem(dims, bc, 5, 0.1, False)
    ref = bbpp.Solver(g).solve_host(b, mask, tol=1e-8, precision=bbpp.FP64)
    x, rep = bbpp.Solver(g).solve_host(b, mask, tol=1e-8, precision=bbpp.FP32_IR)
    assert rep.status == bbpp.CONVERGED and rep.true_rel <= 1.01e-8
    assert rep.iters <= 3 * ref[1].iters + 3 * 50
    # the smallest eigenvalue of L / dL with a solid cell within a few cells of each
    # fluid one is above 1e-2
    assert np.abs(x - ref[0]).max() <= 1e2 * 2e-8 * np.linalg.norm(ref[0])
