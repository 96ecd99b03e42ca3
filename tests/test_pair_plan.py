"""The steps of a pair of FP32 iterations (pair_plan in
bluebottle-3.0_gb300/csrc/bbpp_pair_plan.cuh), compiled for the host: conjugate
gradients' own where its products have digits, one safe step where they have none."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include "bbpp_pair_plan.cuh"
int main() {  // rows of 13 doubles in (the products, fresh, expected), 8 out
  double v[13];
  while (fread(v, 8, 13, stdin) == 13) {
    const bbpp::PairPlan o = bbpp::pair_plan(v, v[11] != 0.0, v[12]);
    const double out[8] = {o.a0, o.b0, o.a1, o.b1, (double)o.steps, (double)o.anew, (double)o.fresh, o.rz};
    fwrite(out, 8, 8, stdout);
  }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    sys.path.insert(0, os.path.join(ROOT, "bluebottle-3.0_gb300"))
    import build
    d = tmp_path_factory.mktemp("pair_plan")
    (d / "p.cu").write_text(SRC)
    try:
        subprocess.run([build.nvcc()] + build.ARCH + ["-O2", "-std=c++17", "-I", build.CSRC, "-o", str(d / "p"),
                                                      str(d / "p.cu")], check=True, capture_output=True)
    except FileNotFoundError:
        pytest.skip("no nvcc")

    def run(prod, fresh, expected):
        v = np.array(list(prod) + [float(fresh), expected], np.float64)
        out = subprocess.run([str(d / "p")], input=v.tobytes(), check=True, capture_output=True).stdout
        a0, b0, a1, b1, steps, anew, nxt, rz = np.frombuffer(out)
        return dict(a0=a0, b0=b0, a1=a1, b1=b1, steps=int(steps), anew=bool(anew), fresh=bool(nxt), rz=rz)
    return run


def operator(n, seed):
    """A symmetric positive definite L with a diagonal that varies, as at walls."""
    rng = np.random.default_rng(seed)
    q = rng.standard_normal((n, n))
    a = q @ q.T / n + np.eye(n)
    return a, np.diag(a).copy()


def products(a, d, z, p):
    r, w = d * z, a @ p
    q, s = w / d, a @ z
    t = a @ q
    rz = r @ z
    return [rz, r @ r - rz, p @ w, z @ w, q @ w, z @ s, z @ t, q @ t, s @ (s / d), s @ (t / d),
            t @ (t / d)]


def cg(a, d, z, p, steps):
    """alpha, beta of each step, and z, p after them."""
    out = []
    for _ in range(steps):
        r, w = d * z, a @ p
        al = (r @ z) / (p @ w)
        z1 = z - al * w / d
        be = (d * z1 @ z1) / (r @ z)
        out.append((al, be))
        z, p = z1, z1 + be * p
    return out, z, p


@pytest.mark.parametrize("seed", range(4))
def test_ordinary_pairs_are_conjugate_gradients(plan, seed):
    a, d = operator(60, seed)
    z = np.random.default_rng(seed + 9).standard_normal(60)
    p, fresh, expected = z.copy(), True, 0.0
    for _ in range(3):
        got = plan(products(a, d, z, p), fresh, expected)
        coefs, z, p = cg(a, d, z, p, 2)
        assert got["steps"] == 2 and not got["fresh"] and got["anew"] == fresh
        np.testing.assert_allclose([got["a0"], got["b0"], got["a1"], got["b1"]], np.ravel(coefs), rtol=1e-9)
        fresh, expected = False, got["rz"]
        assert abs(expected / (d * z @ z) - 1) < 1e-9


def test_nothing_left_after_one_step(plan):
    """p = z an eigenvector of eigenvalue 2 of L (dL = 1), or L the identity: the products are exact, 0 / 0 before."""
    for lam in (2.0, 1.0):
        rz = 4096.0
        prod = [rz, 0.0] + [rz * lam ** k for k in (1, 1, 2, 1, 2, 3, 2, 3, 4)]
        got = plan(prod, True, 0.0)
        assert got["steps"] == 1 and got["fresh"] and got["b0"] == 0.0 and got["a0"] == 1.0 / lam


def test_little_left_after_the_first_or_second_step(plan):
    a, d = operator(40, 1)
    z = np.random.default_rng(2).standard_normal(40)
    prod = products(a, d, z, z)
    (a0, _), = cg(a, d, z, z, 1)[0]
    # (z, w) moved so that the first step leaves a part f of (r,z): 1 - 2 a0 zw / rz + a0^2 qw / rz = f
    for f, fresh in ((2.0 ** -4, False), (2.0 ** -6, False), (2.0 ** -11, True), (-1e-3, True), (0.0, True)):
        moved = list(prod)
        moved[3] = (1 - f + a0 * a0 * moved[4] / moved[0]) * moved[0] / (2 * a0)
        got = plan(moved, True, 0.0)
        assert got["fresh"] == fresh and np.isfinite(got["a0"]) and np.isfinite(got["b0"])
        if f < 2.0 ** -5:
            assert got["steps"] == 1
            assert got["b0"] == 0.0 if fresh else abs(got["b0"] / f - 1) < 1e-6
    # a second step that leaves nothing (two eigenvectors) is left to the next pair
    lam = np.array([1.0, 1.7])
    z = np.array([1.0, 0.8])
    got = plan(products(np.diag(lam), np.ones(2), z, z), True, 0.0)
    assert got["steps"] == 1 and not got["fresh"] and got["b0"] > 0


def test_a_direction_that_is_not_conjugate(plan):
    """An (r,z) that is not the expected one, or a p without curvature: one step along z."""
    a, d = operator(50, 3)
    rng = np.random.default_rng(4)
    z, p = rng.standard_normal(50), rng.standard_normal(50)
    prod = products(a, d, z, p)
    rz = prod[0]
    (want,), _, _ = cg(a, d, z, z, 1)
    for expected, flat in ((rz * 1.3, False), (rz / 1.3, False), (np.nan, False), (0.0, False), (-rz, False),
                           (np.inf, False), (rz, True)):
        bad = list(prod)
        if flat:
            bad[2] = -1e-9
        got = plan(bad, False, expected)
        assert got["steps"] == 1 and got["anew"]
        np.testing.assert_allclose([got["a0"], got["b0"]], want, rtol=1e-12)
    assert not plan(prod, False, rz * 1.01)["anew"]
