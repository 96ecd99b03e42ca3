"""The sum across threads of the FP32 iterations' dot products (sum_floats in
bluebottle-3.0_gb300/csrc/bbpp_dev.cuh), compiled for the host: no less exact
than the FP64 adds that it stands for, over FP32's whole range."""
import math
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdio>
#include <vector>
#include "bbpp_dev.cuh"
int main(int argc, char **argv) {  // rows of 512 floats in, 32 doubles a row out
  std::vector<float> v(512);
  while (fread(v.data(), 4, 512, stdin) == 512)
    for (int lane = 0; lane < 32; lane++) {
      const double s = bbpp::sum_floats(v.data(), 512, lane);
      fwrite(&s, 8, 1, stdout);
    }
}
"""


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    sys.path.insert(0, os.path.join(ROOT, "bluebottle-3.0_gb300"))
    import build
    d = tmp_path_factory.mktemp("sum_floats")
    (d / "s.cu").write_text(SRC)
    try:
        subprocess.run([build.nvcc()] + build.ARCH + ["-O2", "-std=c++17", "-I", build.CSRC, "-o", str(d / "s"),
                                                      str(d / "s.cu")], check=True, capture_output=True)
    except FileNotFoundError:
        pytest.skip("no nvcc")

    def run(v):
        v = np.ascontiguousarray(v, np.float32)
        out = subprocess.run([str(d / "s")], input=v.tobytes(), check=True, capture_output=True).stdout
        return np.frombuffer(out).reshape(len(v), 32)
    return run


def test_no_less_exact_than_fp64(sums):
    rng = np.random.default_rng(1)
    v = rng.standard_normal((400, 512))
    v[100:200] *= np.exp2(rng.integers(-30, 31, (100, 512)))      # spread
    v[200:300, 256:] = -v[200:300, :256] * (1 + 1e-7)             # cancelling
    v[300:] = v[300:] ** 2 * np.exp2(rng.integers(-100, 100, (100, 1)))
    v = v.astype(np.float32)
    got = sums(v)
    for row, g in zip(v, got):
        for lane in range(32):
            x = row[lane::32].astype(np.float64)
            exact, size = math.fsum(x), np.abs(x).sum()
            # half an ulp twice, and 16^2 2^-72 of the magnitudes; sixteen FP64 adds have 15 2^-53 of them
            assert abs(g[lane] - exact) <= 2.0 ** -52 * abs(exact) + 2.0 ** -64 * size


def test_out_of_range(sums):
    big = np.zeros((6, 512), np.float32)
    big[0] = 3e38                                   # a sum that FP32 cannot hold
    big[1] = 3e38
    big[1, 256:] = -3e38
    big[2, 64] = np.inf
    big[3, 64], big[3, 96] = np.inf, -np.inf
    big[4, 64] = np.nan
    big[5] = 1e-45                                  # subnormal
    got = sums(big)
    with np.errstate(invalid="ignore"):
        want = np.array([[row[lane::32].astype(np.float64).sum() for lane in range(32)] for row in big])
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    assert same.all()
