"""The reciprocal of the Poisson kernel's eigenvalues, compiled for the host from the header that the transforms' kernels
use.  Bound: Newton's last step rounds twice (1 - A1 r, then r), so the result lies within two units of FP64 rounding; one
step from an FP32 seed leaves 2^-46."""
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest
from conftest import PKG

CUDA = os.path.dirname(os.path.dirname(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"))

MAIN = r'''
#include "fft.cuh"
#include <cstdio>
int main() {
    double a;
    while (std::fread(&a, 8, 1, stdin) == 1) {
        const double r = mgg::green_reciprocal(a);
        std::fwrite(&r, 8, 1, stdout);
    }
}
'''


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")), reason="no CUDA headers")
def test_reciprocal_is_an_fp64_one(tmp_path):
    src, exe = tmp_path / "r.cpp", tmp_path / "r"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", f"-I{PKG}/csrc", f"-I{CUDA}/include", "-o", str(exe),
                    str(src)], check=True)
    rng = np.random.default_rng(4)
    g = 2 * np.cos(6.28318530718 * np.arange(129) / 256)
    a = (g[rng.integers(0, 129, (3, 4000))].sum(0) - 6)
    a = np.concatenate([a[np.abs(a) > 1e-7], -np.exp(rng.uniform(np.log(1e-7), np.log(12), 2000)), [1.0]])
    r = np.frombuffer(subprocess.run([str(exe)], input=a.tobytes(), capture_output=True, check=True).stdout)
    err = max(abs(Fraction(float(x)) * Fraction(float(y)) - 1) for x, y in zip(a, r))
    assert r.size == a.size and err < Fraction(1, 2 ** 52), float(err)
