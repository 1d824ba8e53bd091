"""The GPU LMS estimator (include/afd_lms.h) against the reference's own
EstimateIr outputs (tests/golden/lms.npz) and the CPU restatement. The GPU
evaluates the reference recursion in blocks of 128 samples, which changes
only the order of floating-point additions: bar 1e-10 relative L2."""
import os

import numpy as np
import pytest

import lms_oracle

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
TOL = 1e-10


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("name", ["fir4", "odd", "short_out", "room"])
def test_gpu_equals_reference_outputs(pkg, name):
    g = np.load(os.path.join(HERE, "golden", "lms.npz"))
    N, mu = g[name + "_meta"]
    got = pkg.lms.EstimateIr(g[name + "_x"], g[name + "_y"], int(N), float(mu))
    assert rel(got, g[name + "_w"]) < TOL


def test_gpu_many_tap_chunks_equals_restatement(pkg):
    """More taps than one CTA of the y0 pass handles (2048), several blocks."""
    rng = np.random.default_rng(9)
    N, steps = 3000, 700
    x = rng.standard_normal(steps)
    h = rng.standard_normal(N) * np.exp(-np.arange(N) / 300.0)
    d = np.convolve(x, h)[:steps]
    want = lms_oracle.estimate(x, d, N, 2e-4, epochs=2)
    got = pkg.lms.estimate_ir(x, d, N, 2e-4, epochs=2)
    assert rel(got, want) < TOL


def test_gpu_identifies_a_known_response(pkg):
    """Noise-free identification of a 200-tap response from 20000 samples of
    white noise: the reference's 16 passes converge to it."""
    rng = np.random.default_rng(10)
    h = rng.standard_normal(200) * np.exp(-np.arange(200) / 40.0)
    x = rng.standard_normal(20000)
    d = np.convolve(x, h)[:20000]
    w = pkg.lms.EstimateIr(x, d, 200, 1e-3)
    assert rel(w, h) < 1e-6


# edges of the 512-sample blocks and 32-tap strides, unequal lengths, more tap
# tiles than CTAs (70000 taps), more blocks than one segment of inverses holds
# (400000 samples); the same bar as above, the recursion being reassociated
# the same way whatever the sizes
@pytest.mark.parametrize("taps,nx,nd,epochs", [
    (1, 1, 1, 1), (1, 700, 513, 3), (31, 511, 511, 2), (32, 512, 600, 2), (33, 513, 1025, 1), (224, 1030, 1024, 16),
    (4737, 1500, 1300, 2), (70000, 600, 600, 3), (9, 400000, 400000, 2)])
def test_gpu_block_and_tile_edges(pkg, taps, nx, nd, epochs):
    rng = np.random.default_rng(taps + nx)
    x, d = rng.standard_normal(nx), rng.standard_normal(nd)
    mu = min(2e-3, 0.05 / taps)
    want = lms_oracle.estimate(x, d, taps, mu, epochs=epochs)
    got = pkg.lms.estimate_ir(x, d, taps, mu, epochs=epochs)
    assert rel(got, want) < TOL


def test_gpu_nothing_to_do_and_repeats(pkg):
    """No samples or no pass leave zeros; a call gives the same bits again
    after other sizes have used the kept workspace, also from two threads."""
    from concurrent.futures import ThreadPoolExecutor
    rng = np.random.default_rng(4)
    x, d = rng.standard_normal(2000), rng.standard_normal(2000)
    assert not pkg.lms.estimate_ir(x[:0], d, 7, 1e-3).any()
    assert not pkg.lms.estimate_ir(x, d, 7, 1e-3, epochs=0).any()
    first = pkg.lms.estimate_ir(x, d, 300, 1e-4, epochs=2)
    pkg.lms.estimate_ir(x[:900], d, 5000, 1e-6, epochs=1)
    with ThreadPoolExecutor(2) as pool:
        again = list(pool.map(lambda n: pkg.lms.estimate_ir(x, d, n, 1e-4, epochs=2), [300, 301, 300, 40]))
    assert np.array_equal(first, again[0]) and np.array_equal(first, again[2])
