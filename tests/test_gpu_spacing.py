"""Checkpoints further apart than any solve is long: none is met, in every form."""
import numpy as np
import pytest

import bbpp
from bbpp import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["resident", "kernels"])
@pytest.mark.parametrize("precision", [bbpp.FP64, bbpp.FP32_IR])
@pytest.mark.parametrize("replace_every", [70000, 2 ** 30, 2 ** 31 - 1])
def test_no_checkpoint_is_met(bbpp_lib, monkeypatch, form, precision, replace_every):
    monkeypatch.setenv("BBPP_PERSIST", "1" if form == "resident" else "0")
    g, mask, rhs, _ = problems.make_problem("C2", n=32)
    kw = dict(tol=1e-6, precision=precision, max_iter=400)
    x, rep = bbpp.Solver(g).solve_host(rhs, mask, replace_every=replace_every, **kw)
    y, rep2 = bbpp.Solver(g).solve_host(rhs, mask, replace_every=500, **kw)
    assert rep.status == rep2.status == bbpp.CONVERGED
    assert rep.iters == rep2.iters and np.array_equal(x, y)
