"""The GPU LMS estimator at the limits of its block form (explicit inverses of 512
samples): step sizes near and beyond the stable range and values that are not
finite, against the CPU restatement of the sample-by-sample recursion.

Tolerance: the recursion reassociated is exact up to the order of additions; a
deviation of 2^-53 per operation is carried on by the recursion itself, near the
stability limit without decay, over 12000 samples and a few thousand
operations each: 1e-10, the bar of all LMS tests."""
import numpy as np
import pytest

import lms_oracle

pytestmark = pytest.mark.gpu
TOL = 1e-10


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


# mu x taps x power (the stable range of white noise ends near 1); 24 blocks;
# correlated inputs reach their limit sooner
@pytest.mark.parametrize("level,kind", [(0.7, "white"), (0.8, "white"), (0.9, "white"), (0.6, "sine"), (0.95, "sine"),
                                        (0.45, "bursts")])
def test_near_the_stability_limit(pkg, level, kind):
    rng = np.random.default_rng(3)
    N, n = 150, 12000
    t = np.arange(n)
    x = {"white": rng.standard_normal(n), "sine": np.sin(0.05 * t) + 0.01 * rng.standard_normal(n),
         "bursts": rng.standard_normal(n) * (0.01 + (t // 700 % 3 == 1))}[kind]
    d = np.convolve(x, rng.standard_normal(N) * np.exp(-np.arange(N) / 30.0))[:n] + 0.01 * rng.standard_normal(n)
    power = np.mean(x * x) if kind != "bursts" else 1.0
    mu = level / (N * power)
    want = lms_oracle.estimate(x, d, N, mu, epochs=1)
    assert np.isfinite(want).all() and np.abs(want).max() < 1e3
    assert rel(pkg.lms.estimate_ir(x, d, N, mu, epochs=1), want) < TOL


# few taps near the limit: within a block an error grows by several orders before
# it falls again, and the weights converge or stay small all the same. The bar is
# that of the other tests; by the inverses of 512 samples 1e-9 to 1e-7
@pytest.mark.parametrize("N,level,seed", [(2, 0.8, 4), (4, 0.85, 1), (4, 0.85, 2), (4, 0.85, 3), (8, 0.9, 4)])
def test_errors_that_grow_within_a_block(pkg, N, level, seed):
    rng = np.random.default_rng([N, seed])
    n = 2600
    x = rng.standard_normal(n)
    d = np.convolve(x, [1, 0.5, 0.2])[:n] + 0.01 * rng.standard_normal(n)
    mu = level / (N * np.mean(x * x))
    want = lms_oracle.estimate(x, d, N, mu, epochs=1)
    assert np.abs(want).max() < 1e4
    assert rel(pkg.lms.estimate_ir(x, d, N, mu, epochs=1), want) < TOL


def test_silence_stays_silent_at_any_step_size(pkg):
    """No output to identify: the weights stay zero although an error would grow
    beyond every bound within a block."""
    rng = np.random.default_rng(4)
    x = 1.0 + 0.1 * rng.standard_normal(1500)
    assert not pkg.lms.estimate_ir(x, np.zeros(1500), 20, 1.0, epochs=2).any()


@pytest.mark.parametrize("N,n,epochs", [(1, 512, 1), (3, 515, 1), (40, 300, 2)])
def test_growth_that_stays_in_range(pkg, N, n, epochs):
    """An unstable step size with errors so small that the recursion ends within
    the range of FP64, where one started at 1 would have left it: the values of
    the restatement."""
    rng = np.random.default_rng(N)
    x = 1.0 + 0.01 * rng.standard_normal(n)
    d = 1e-290 * rng.standard_normal(n)
    mu = 3.0 / N
    want = lms_oracle.estimate(x, d, N, mu, epochs=epochs)
    assert np.isfinite(want).all() and np.abs(want).max() > 1e-100
    assert rel(pkg.lms.estimate_ir(x, d, N, mu, epochs=epochs) / np.abs(want).max(), want / np.abs(want).max()) < TOL


# an output sample that is not finite: what comes before it in its block is
# still right; with it in the last sample, the weights are its own update
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("n", [40, 513, 1000])
def test_output_that_is_not_finite(pkg, bad, n):
    rng = np.random.default_rng(5)
    N = 24
    x, d = rng.standard_normal(n), rng.standard_normal(n)
    d[-1] = bad
    with np.errstate(invalid="ignore"):
        want = lms_oracle.estimate(x, d, N, 1e-2, epochs=1)
    assert np.array_equal(pkg.lms.estimate_ir(x, d, N, 1e-2, epochs=1), want, equal_nan=True)


def test_input_that_is_not_finite(pkg):
    """From an input sample that is not finite on, no weight is a number."""
    rng = np.random.default_rng(6)
    for bad in (np.inf, np.nan):
        x, d = rng.standard_normal(900), rng.standard_normal(900)
        x[700] = bad
        assert np.isnan(pkg.lms.estimate_ir(x, d, 30, 1e-3, epochs=1)).all()
