"""The FP64 method keeps every search direction, as the reference does: with a
residual replaced in every iteration, a beta of more than four (the first steps
on a smooth right-hand side with spheres) is the iteration's own."""
import numpy as np
import pytest

import bbpp
from bbpp import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [48, 64])
@pytest.mark.parametrize("resident", ["0", "1"])
def test_fp64_keeps_its_direction(bbpp_lib, orc, monkeypatch, n, resident):
    monkeypatch.setenv("BBPP_PERSIST", resident)
    g, mask, rhs, _ = problems.make_problem("C2", n=n)
    s = bbpp.Solver(g)
    s.set_trace(8)
    x, rep = s.solve_host(rhs, mask, tol=1e-10, replace_every=1)
    a, b = s.trace()
    xo, res = orc.pcg(orc.from_tuple(g.as_tuple()), rhs, mask, tol=1e-10, replace_every=1, trace=8)
    assert res["beta"][:8].max() > 4.0  # the case that this is about
    # alpha and beta of the first iterations: a residual formed from x carries 2^-53 |x| / |r| of the right-hand
    # side's scale, 1e-13 here, and eight steps amplify it by their betas' product, below 1e4
    assert np.all(np.abs(a / res["alpha"][:8] - 1) <= 1e-9)
    assert np.all(np.abs(b / res["beta"][:8] - 1) <= 1e-9)
    assert rep.status == bbpp.CONVERGED and abs(rep.iters - res["iters"]) <= 2
