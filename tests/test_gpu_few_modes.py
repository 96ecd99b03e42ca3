"""Mixed-precision solves whose right-hand side lies in few eigenvectors, or that
one step solves: the expansions that a step's coefficients come from cancel
there.  Against the solution in closed form, within the iterations that the noise
FP32 leaves of such a residual takes (a uniform right-hand side's, below 200)."""
import numpy as np
import pytest

import bbpp
from bbpp import problems

pytestmark = pytest.mark.gpu


def modes(n, names):
    """The sum of the named eigenvectors of the periodic Laplacian on n^3 cells and the solution for it."""
    k, j, i = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    th = 2 * np.pi / n
    table = {
        "checker": ([(n // 2,) * 3], 1.0 - 2.0 * ((i + j + k) % 2)),
        "planes_z": ([(0, 0, n // 2)], 1.0 - 2.0 * (k % 2)),
        "planes_x": ([(n // 2, 0, 0)], 1.0 - 2.0 * (i % 2)),
        "low": ([(1, 2, 3)], np.sin(th * i) * np.sin(2 * th * j) * np.sin(3 * th * k)),
        "middle": ([(5, 7, 0)], np.sin(5 * th * i) * np.sin(7 * th * j)),
        "rough": ([(n // 2 - 1, 0, 0)], np.sin((n // 2 - 1) * th * i)),
        "quarter": ([(n // 4, 0, 0)], np.sin((n // 4) * th * i)),
        "wave": ([(0, 0, 2)], np.sin(2 * th * k)),
    }
    b, x = np.zeros((n,) * 3), np.zeros((n,) * 3)
    for name in names:
        (m,), f = table[name]
        lam = sum(2.0 - 2.0 * np.cos(th * q) for q in m) * n * n
        b += f
        x += f / lam
    return b, x


def solve(monkeypatch, form, g, b, mask, tol):
    """form: pair, fused, fused_ws, two (search + update kernels) or resident."""
    if form == "fused_ws":
        monkeypatch.setenv("BBPP_FUSED_WS", "1")
    monkeypatch.setenv("BBPP_PERSIST", "1" if form == "resident" else "0")
    monkeypatch.setenv("BBPP_PAIR", "1" if form == "pair" else "0")
    s = bbpp.Solver(g)
    if form == "two":
        s.set_fused(False)
    x, rep = s.solve_host(b, mask, tol=tol, precision=bbpp.FP32_IR, max_iter=200,
                          ok=(bbpp.CONVERGED, bbpp.MAX_ITER, bbpp.NAN))
    return x, rep


FORMS = [("pair", 48), ("pair", 64), ("fused", 64), ("fused_ws", 64), ("two", 48), ("two", 64),
         ("resident", 48), ("resident", 64)]


@pytest.mark.parametrize("tol", [1e-4, 1e-6, 1e-8, 1e-10])
@pytest.mark.parametrize("names", [("checker",), ("planes_z",), ("planes_x",), ("low",), ("middle",), ("rough",),
                                   ("quarter",), ("checker", "wave"), ("wave", "rough")], ids="+".join)
@pytest.mark.parametrize("form,n", FORMS)
def test_few_modes(bbpp_lib, monkeypatch, form, n, names, tol):
    g = bbpp.Grid.make(n, n, n, 1.0 / n, 1.0 / n, 1.0 / n, problems.bc_tuple("ppp"))
    b, xe = modes(n, names)
    x, rep = solve(monkeypatch, form, g, b, None, tol)
    assert rep.status == bbpp.CONVERGED and rep.true_rel <= 1.01 * tol and np.isfinite(x).all()
    # both within tol of a zero residual: the error is below tol times the condition number of the scaled operator
    # on the fields of mean zero, (n / pi)^2 (the mean itself is free)
    x -= x.mean()
    assert np.linalg.norm(x - xe) <= (n / np.pi) ** 2 * tol * np.linalg.norm(xe)


def test_checkerboard_on_the_default_path(bbpp_lib):
    n = 192
    g = bbpp.Grid.make(n, n, n, 1.0 / n, 1.0 / n, 1.0 / n, problems.bc_tuple("ppp"))
    b, xe = modes(n, ["checker"])
    for scale in (1.0, 3.7e-3, 1.3e5):
        x, rep = bbpp.Solver(g).solve_host(scale * b, None, tol=1e-8, precision=bbpp.FP32_IR,
                                           ok=(bbpp.CONVERGED, bbpp.NAN))
        assert rep.status == bbpp.CONVERGED and rep.iters <= 2 and np.isfinite(x).all()
        # one eigenvector of eigenvalue 2 of the scaled operator, the largest: the error is the residual's tol
        assert np.abs(x - x.mean() - scale * xe).max() <= 1e-8 * scale * np.abs(xe).max() * np.sqrt(n ** 3)


@pytest.mark.parametrize("form", ["pair", "fused", "resident"])
@pytest.mark.parametrize("bc", ["ppp", "ppn", "nnn"])
def test_isolated_fluid_cells(bbpp_lib, monkeypatch, form, bc):
    """No fluid cell has a fluid neighbour: the operator is its diagonal, one step solves it.  (Against walls the
    diagonal differs, and Jacobi's preconditioner takes it out.)"""
    n = 64
    g = bbpp.Grid.make(n, n, n, 1.0 / n, 1.0 / n, 1.0 / n, problems.bc_tuple(bc))
    k, j, i = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    mask = ((i + j + k) % 2).astype(np.uint8)
    b = np.random.default_rng(3).uniform(-1, 1, g.shape)
    b[mask == 1] = 0
    diag = np.zeros(g.shape)
    for axis, c in enumerate("zyx"):
        diag += 2.0
        if bc[2 - axis] == "n":
            for e in (0, n - 1):
                diag[tuple(e if a == axis else slice(None) for a in range(3))] -= 1.0
    xe = b / (diag * n * n)
    x, rep = solve(monkeypatch, form, g, b, mask, 1e-8)
    # FP32 leaves 6e-8 of the residual after one step, so a second and a confirmation's third
    assert rep.status == bbpp.CONVERGED and rep.iters <= 4
    assert np.linalg.norm(x - xe) <= 4 * 1e-8 * np.linalg.norm(xe)


@pytest.mark.parametrize("dims,bc", [((64, 45, 30), "ppn"), ((48, 40, 33), "nnn"), ((256, 29, 20), "ppp")])
def test_pairs_that_lose_their_direction(bbpp_lib, monkeypatch, dims, bc):
    """Every sixth pair goes along z instead of p (a test hook): one step, and
    conjugate gradients from there.  Each stretch reduces the error, so the solve
    converges, if later than one that keeps its directions."""
    monkeypatch.setenv("BBPP_PERSIST", "0")
    nx, ny, nz = dims
    g = bbpp.Grid.make(nx, ny, nz, 1.0 / nx, 1.0 / ny, 1.0 / nz, problems.bc_tuple(bc))
    rng = np.random.default_rng(7)
    mask = (rng.random(g.shape) < 0.05).astype(np.uint8)
    b = rng.uniform(-1, 1, g.shape)
    b[mask == 1] = 0
    b[mask == 0] -= b[mask == 0].mean()
    kw = dict(tol=1e-8, precision=bbpp.FP32_IR)
    s = bbpp.Solver(g)
    x0, rep0 = s.solve_host(b, mask, **kw)
    assert bbpp.lib().bbpp_debug_wait(s.handle, 0, 6) == 0
    x, rep = s.solve_host(b, mask, **kw)
    assert rep.status == bbpp.CONVERGED and rep.true_rel <= 1.01e-8
    assert rep.iters > rep0.iters
    # both within tol of a zero residual, the condition number below (2 n / pi)^2
    assert np.abs(x - x0).max() <= (2 * max(dims) / np.pi) ** 2 * 1e-8 * np.abs(x0).max()
