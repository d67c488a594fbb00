"""The kernels' sums in triples of floats (csrc/vg_internal.cuh) lose no more than
the sums in FP64 that they stand for: against exactly rounded sums, one rounding
and n^2 2^-72 of the sum of magnitudes."""
import math
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    from vortegrid_gb300 import build
    tmp = tmp_path_factory.mktemp("sums")
    exe = str(tmp / "sums")
    subprocess.check_call([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                           build.CSRC, os.path.join(ROOT, "tests", "cpp", "sums.cu"), "-o", exe])

    def run(v):
        with open(tmp / "in.bin", "wb") as f:
            np.array(v.shape, np.int32).tofile(f)
            v.tofile(f)
        subprocess.check_call([exe, str(tmp / "in.bin"), str(tmp / "out.bin")])
        return np.fromfile(tmp / "out.bin", np.float64).reshape(-1, 3)
    return run


@pytest.mark.parametrize("n", [1, 2, 41, 1000])
@pytest.mark.parametrize("spread", [0.0, 6.0])
def test_no_less_than_fp64(sums, n, spread):
    """spread: the values' magnitudes over 10^+-spread."""
    rng = np.random.default_rng(n)
    v = (rng.normal(0, 1, (300, n)) * 10.0 ** rng.uniform(-spread, spread, (300, n))).astype(np.float32)
    got = sums(v)
    for row, (s, q, _) in zip(v.astype(np.float64), got):
        exact, squares = math.fsum(row), math.fsum(row * row)  # squares of floats are exact in float64
        lost = n * n * 2.0 ** -72
        assert abs(s - exact) <= 2.0 ** -52 * abs(exact) + lost * math.fsum(abs(row))
        assert abs(q - squares) <= (2.0 ** -52 + lost) * squares


def test_range_of_squares(sums):
    """Sums that squares outside the range of floats may have spoilt are told from
    the others, among them those of zeros alone."""
    rows = {"zeros": (0.0, 0.0, True), "minus zero": (-0.0, 0.0, True), "ones": (1.0, 1.0, True),
            "zeros and ones": (0.0, 1.0, True), "small": (0.0, 1e-20, False), "subnormal": (0.0, 1e-40, False),
            "large": (1.0, 1e19, False), "infinite": (0.0, np.inf, False), "not a number": (0.0, np.nan, False)}
    v = np.zeros((len(rows), 41), np.float32)
    for k, (a, b, _) in enumerate(rows.values()):
        v[k] = a
        v[k, 20] = b
    assert [bool(x) for x in sums(v)[:, 2]] == [r[2] for r in rows.values()]
