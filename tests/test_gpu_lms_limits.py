"""The GPU LMS estimator at the limits of its block form (explicit inverses of 512
samples): values that are not finite, against the CPU restatement of the
sample-by-sample recursion."""
import numpy as np
import pytest

import lms_oracle

pytestmark = pytest.mark.gpu


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
