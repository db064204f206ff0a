"""The FP64 sweep's reciprocal, one MUFU approximation and one third-order step, against IEEE division.

The approximation works on the upper 32 bits of its operand and of its result: two truncations of 2^-20 each, and
as much again for the approximation itself, is |e| < 2^-18.  The step leaves out e^3 < 2^-54, half a unit in the last
place at most, and its last operation rounds once more: less than one unit from 1/x, so that it is IEEE division's
result or a neighbour of it."""
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def reciprocals(tmp_path_factory):
    d = tmp_path_factory.mktemp("rcp")
    rng = np.random.default_rng(1)
    bits = rng.integers(0, 1 << 52, 1 << 20, dtype=np.uint64)
    bits[: 1 << 16] |= np.uint64(0xFFFFFFFF)  # what the approximation does not see, at its largest
    bits[1 << 16: 1 << 17] &= np.uint64(0xFFFFF00000000)
    mant = np.concatenate([bits, np.arange(1 << 12, dtype=np.uint64), np.uint64((1 << 52) - 1) - np.arange(1 << 12, dtype=np.uint64)])
    expo = rng.integers(1023 - 1000, 1023 + 1000, mant.size).astype(np.uint64)
    expo[::2] = 1023  # one binade in detail
    x = ((expo << np.uint64(52)) | mant).view(np.float64)
    x[1::7] *= -1.0
    exe = str(d / "probe")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                    os.path.join(ROOT, "tcsem_fdtd_gb300", "csrc"), "-o", exe, os.path.join(ROOT, "tests", "rcp64_probe.cu")],
                   check=True)
    x.tofile(d / "x")
    subprocess.run([exe, str(d / "x"), str(d / "r")], check=True)
    return x, np.fromfile(d / "r")


def test_reciprocal_is_ieee_division_or_its_neighbour(reciprocals):
    x, r = reciprocals
    ulp = np.abs(r.view(np.int64) - (1.0 / x).view(np.int64))
    assert int(ulp.max()) <= 1


def test_reciprocal_is_within_a_unit_of_the_exact_value(reciprocals):
    x, r = reciprocals
    pick = np.concatenate([np.arange(0, x.size, 97), np.arange(x.size - (1 << 13), x.size)])
    worst = max(abs(Fraction(float(r[q])) - 1 / Fraction(float(x[q]))) / Fraction(float(np.spacing(abs(1.0 / x[q])))) for q in pick)
    print("largest error in units in the last place:", float(worst))
    assert worst < 1
