"""The form of the FP32 iteration that a context is asked for is the one that
runs: by its kernels' names in the kernel statistics, and by what a wait that
runs out in it does to a solve."""
import numpy as np
import pytest

import bbpp
from bbpp import problems

pytestmark = pytest.mark.gpu

FORMS = {"default": {"pair_f32", "dots_f32"}, "fused": {"fused_f32"}, "two": {"search_spmv_f32", "update_f32"},
         "ws0": {"fused_f32"}, "ws1": {"fused_f32"}}


def make(monkeypatch, form):
    if form.startswith("ws"):
        monkeypatch.setenv("BBPP_FUSED_WS", form[2])
    g, mask, rhs, _ = problems.make_problem("C3", n=64)
    s = bbpp.Solver(g)
    if form in ("fused", "two"):
        s.set_fused(form == "fused")
    return s, mask, rhs


@pytest.mark.parametrize("form", FORMS)
def test_a_form_runs_its_kernels(bbpp_lib, monkeypatch, form):
    s, mask, rhs = make(monkeypatch, form)
    s.set_profiling(True)  # kernel by kernel: the default is then the pairs
    s.solve_host(rhs, mask, tol=1e-8, precision=bbpp.FP32_IR)
    kinds = {k[0] for k in s.kernel_stats()}
    every = set().union(*FORMS.values())
    assert kinds & every == FORMS[form]


@pytest.mark.parametrize("form", FORMS)
def test_a_form_reports_its_wait(bbpp_lib, monkeypatch, form):
    """Without profiling: the resident iteration by default, else the kernels asked for."""
    s, mask, rhs = make(monkeypatch, form)
    L = bbpp.lib()
    assert L.bbpp_debug_wait(s.handle, 2_000_000, 1) == 0
    x, rep = s.solve_host(rhs, mask, tol=1e-8, precision=bbpp.FP32_IR, ok=(bbpp.WAIT_TIMEOUT,))
    assert rep.status == bbpp.WAIT_TIMEOUT
    assert L.bbpp_debug_wait(s.handle, 0, 0) == 0
    x, rep = s.solve_host(rhs, mask, tol=1e-8, precision=bbpp.FP32_IR)
    assert rep.status == bbpp.CONVERGED and rep.true_rel <= 1.01e-8


@pytest.mark.parametrize("form", ["fused", "two"])
def test_a_form_asked_for_is_not_the_default(bbpp_lib, monkeypatch, form):
    """Other kernels, other roundings: not the default's bits."""
    s, mask, rhs = make(monkeypatch, form)
    x, rep = s.solve_host(rhs, mask, tol=1e-8, precision=bbpp.FP32_IR)
    y, rep2 = make(monkeypatch, "default")[0].solve_host(rhs, mask, tol=1e-8, precision=bbpp.FP32_IR)
    assert not np.array_equal(x, y) and np.abs(x - y).max() <= 1e-5 * np.abs(y).max()


@pytest.mark.parametrize("form,dims", [("pair", (64, 45, 30)), ("pair", (64, 64, 64)), ("fused", (64, 64, 64))])
def test_no_memory_for_a_form(bbpp_lib, monkeypatch, form, dims):
    """The vectors that only the pairs or the fused iteration need cannot be had (the
    host's fake of the failing call): the solve takes the search and update kernels,
    which need none, to the same bits; with memory again, the form itself."""
    monkeypatch.setenv("BBPP_PERSIST", "0")
    if form == "fused":
        monkeypatch.setenv("BBPP_PAIR", "0")
    nx, ny, nz = dims
    g = bbpp.Grid.make(nx, ny, nz, 1.0 / nx, 1.0 / ny, 1.0 / nz, problems.bc_tuple("ppn"))
    rng = np.random.default_rng(1)
    b = rng.uniform(-1, 1, g.shape)
    b -= b.mean()
    kw = dict(tol=1e-8, precision=bbpp.FP32_IR)
    s, s2 = bbpp.Solver(g), bbpp.Solver(g)
    s2.set_fused(False)
    x2, _ = s2.solve_host(b, None, **kw)
    L = bbpp.lib()
    assert L.bbpp_debug_wait(s.handle, 0, 4) == 0
    x, rep = s.solve_host(b, None, **kw)
    assert rep.status == bbpp.CONVERGED and np.array_equal(x, x2)
    assert L.bbpp_debug_wait(s.handle, 0, 0) == 0
    x, rep = s.solve_host(b, None, **kw)
    assert rep.status == bbpp.CONVERGED and not np.array_equal(x, x2)


def test_a_checkpoint_every_iteration_goes_one_by_one(bbpp_lib, monkeypatch):
    """Neither a pair nor a resident launch has more than one iteration to do then."""
    s, mask, rhs = make(monkeypatch, "default")
    x, _ = s.solve_host(rhs, mask, tol=1e-8, precision=bbpp.FP32_IR, replace_every=1)
    s.set_profiling(True)
    y, _ = s.solve_host(rhs, mask, tol=1e-8, precision=bbpp.FP32_IR, replace_every=1)
    kinds = {k[0] for k in s.kernel_stats()}
    assert "fused_f32" in kinds and not kinds & FORMS["default"]
    assert np.array_equal(x, y)  # without profiling the same kernels
