"""The FP64 root of the plain path's cells, seeded by Newton's method in FP32, compiled for the host from the header that
the sweeps use, against the root in exact arithmetic.

A value that comes back (NaN sends the cell to the closed form) is the largest root to FP64 rounding: f is rounded to a few
2^-53 of its largest term, at most 9 u^3 here, and divided by a slope of at least u^2, so 1e-14 of the root.  The cases run
down to a double root (slope 0), where an FP32 seed is off by far more than two chord steps mend, and over the range of
values, down to where FP32 underflows."""
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest
from conftest import PKG

CUDA = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))
pytestmark = pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")),
                                reason="no CUDA headers")

MAIN = r'''
#include "roots.cuh"
#include <cstdio>
int main(int argc, char** argv) {
    double a[3];
    while (std::fread(a, 8, 3, stdin) == 3) {
        const double u = argc > 1 ? mgg::root_from<true>((float)a[0], a[1], a[2])
                                  : mgg::root_from<false>((float)a[0], a[1], a[2]);
        std::fwrite(&u, 8, 1, stdout);
    }
}
'''


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("roots")
    (d / "r.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", f"-I{PKG}/csrc", f"-I{CUDA}/include", "-o",
                    str(d / "r"), str(d / "r.cpp")], check=True)
    return str(d / "r")


def relative_error(u, P, Q, power):
    """(u - root) / root, one exact Newton step from u (quadratic: the error's square is far below the bound)."""
    u, P, Q = Fraction(u), Fraction(P), Fraction(Q)
    f, fp = u ** power + P * u + Q, power * u ** (power - 1) + P
    return float(f / fp / u)


# slope: f' at the root over u^2 (u^3); below 2 (3) the cubic (quartic) has Q > 0
@pytest.mark.parametrize("slope", [1e-3, 4e-3, 1e-2, 0.1, 0.5, 0.9, 1.1, 1.5, 2.0, 3.0, 10.0, 1e4])
@pytest.mark.parametrize("power", [3, 4])
def test_root_is_fp64_or_left_to_the_closed_form(exe, power, slope):
    rng = np.random.default_rng(int(1000 * slope) + power)
    n = 400
    root = np.exp(rng.uniform(np.log(1e-16), np.log(1e3), n))
    root[: n // 2] = np.exp(rng.uniform(np.log(1e-6), np.log(10), n // 2))
    P = (slope - power) * root ** (power - 1)
    Q = -(root ** power + P * root)
    start = root * np.exp(rng.uniform(-0.1, 0.3, n))
    got = np.frombuffer(subprocess.run([exe] + ["4"] * (power == 4), input=np.stack([start, P, Q], 1).tobytes(),
                                       capture_output=True, check=True).stdout)
    assert got.size == n
    for u, p, q, r in zip(got, P, Q, root):
        if u == u:
            assert abs(u / r - 1) < 0.5
            assert abs(relative_error(u, p, q, power)) < 1e-14, (u, r, p, q)
    if slope >= power - 1:   # Q <= 0, the common cells: they do not need the closed form
        assert np.mean(np.isnan(got[: n // 2])) < 0.05
