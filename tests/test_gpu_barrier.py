"""The grid barrier of the resident step and of the LMS recursion (sync.cuh) gives
up at its 2 s limit when a block is missing, tells every thread and the host, lets
copies in flight land, and leaves the context usable (afd_barrier_selftest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_barrier_gives_up_and_reports(pkg):
    gave_up, waited = pkg.afd.barrier_selftest(complete=False)
    assert gave_up and 2.0 <= waited < 4.0
    gave_up, waited = pkg.afd.barrier_selftest(complete=True)
    assert not gave_up and waited < 0.1
    # kernels that use it still run
    sim = pkg.Simulation(mode=1)
    sim.SetMinSize(0.3, 0.3, 0.3)
    sim.AddSourceCell((5, 5, 5), np.ones(4, np.float32))
    sim.AddMicCell((8, 8, 8))
    sim.Run(20)
    assert np.all(np.isfinite(sim.mics())) and np.any(sim.mics() != 0)
    sim.close()
    x = np.random.default_rng(0).standard_normal(900)
    assert np.isfinite(pkg.lms.estimate_ir(x, x, 20, 1e-3, epochs=1)).all()
    with pytest.raises(pkg.AfdError):
        pkg.afd.barrier_selftest(complete=True, device=99)
