"""The FP64 step's own exponential, reciprocal and logarithm (tpord_f64.cuh)
against long double, over the arguments the step forms and at their ends.

Bounds, in units of u = 2^-53 of the result:
 2^x    the table's rounding and the last FMA's, 1 each, and 2^-58.5 of
        truncation: 2.1; without a trend at the ends of the polynomial's interval
        (the mean over the table's 256 entries, whose roundings' mean is below 0.06,
        within 0.1);
 1/x    the last FMA's rounding, the correction's error being 2^-60: 1.05;
 log2   absolute: the table's rounding times log2 e (1.45) and the truncation of
        ln(1 + d), plus the product's and the last FMA's roundings: 1.7 + 1.1 |log2 x|."""
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    from lqt1_gb300 import build
    d = tmp_path_factory.mktemp("math")
    exe = str(d / "step_math")
    r = subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-O3", "-I", build.CSRC,
                        os.path.join(ROOT, "tests", "cpp", "step_math.cu"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(op, x):
        np.asarray(x, np.float64).tofile(d / "x")
        assert subprocess.run([exe, op, str(d / "x"), str(d / "y")]).returncode == 0
        return np.fromfile(d / "y")
    return run


def wide(x):
    return np.asarray(x, np.float64).astype(np.longdouble)


def test_exponential(evaluate):
    rng = np.random.default_rng(0)
    x = np.concatenate([rng.uniform(-99.9, 99.9, 200000), rng.uniform(-2, 2, 200000), [0.0, 1.0, -1.0, 1e-20, -1e-300]])
    err = (wide(evaluate("ex2", x)) / np.exp2(wide(x)) - 1).astype(np.float64) / U
    assert np.abs(err).max() <= 2.1
    for side in (-1, 1):
        # next to the ends of every table entry's interval, at many places
        j = np.repeat(np.arange(256), 200)
        x = (j + side * (0.5 - 1e-4 * rng.uniform(0, 1, j.size))) / 256 + rng.integers(-40, 40, j.size)
        err = (wide(evaluate("ex2", x)) / np.exp2(wide(x)) - 1).astype(np.float64) / U
        assert abs(err.mean()) <= 0.1
    ends = evaluate("ex2", [2000.0, -2000.0, 1e300, -1e300, np.inf, -np.inf, np.nan, -np.nan])
    np.testing.assert_array_equal(ends, [2.0 ** 100, 2.0 ** -100] * 3 + [np.nan] * 2)


def test_reciprocal(evaluate):
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(1, 2, 200000), np.exp(rng.uniform(-600, 600, 200000)), -np.exp(rng.uniform(-5, 5, 1000)),
                        [1.0, 2.0, 3.0, 1e-60, 1e60]])
    err = (wide(evaluate("rcp", x)) * wide(x) - 1).astype(np.float64) / U
    assert np.abs(err).max() <= 1.05


def test_logarithm(evaluate):
    rng = np.random.default_rng(2)
    x = np.concatenate([np.exp(rng.uniform(-60, 60, 200000)), rng.uniform(0.5, 2.0, 200000), 2.0 ** np.arange(-40.0, 41),
                        1 + rng.uniform(-1e-3, 1e-3, 1000)])
    ref = np.log2(wide(x))
    err = np.abs(wide(evaluate("lg2", x)) - ref).astype(np.float64) / U
    assert np.all(err <= 1.7 + 1.1 * np.abs(ref.astype(np.float64)))
    ends = evaluate("lg2", [0.0, -0.0, 1e-310, np.inf, -1.0, -np.inf, np.nan])
    np.testing.assert_array_equal(ends, [-np.inf] * 3 + [np.inf] + [np.nan] * 3)
