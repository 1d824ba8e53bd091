"""The device memory that the LMS estimator keeps between calls: bounded, and given
back on request (afd_lms_release) or when another allocation needs it."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


def test_kept_memory_is_bounded_and_given_back(pkg):
    import torch
    rng = np.random.default_rng(1)
    x = rng.standard_normal(450000)  # more blocks than one segment of inverses
    torch.cuda.synchronize()
    pkg.lms.estimate_ir(x[:600], x[:600], 4, 1e-3, epochs=1)  # the kernels' own memory
    pkg.lms.release()
    before = torch.cuda.mem_get_info()[0]
    first = pkg.lms.estimate_ir(x, x, 12, 1e-3, epochs=1)
    kept = before - torch.cuda.mem_get_info()[0]
    assert 100 * MB < kept <= 1100 * MB
    pkg.lms.release()
    assert before - torch.cuda.mem_get_info()[0] < 40 * MB
    # a call after it, and others while memory is given back, are not disturbed
    assert np.array_equal(pkg.lms.estimate_ir(x, x, 12, 1e-3, epochs=1), first)
    with ThreadPoolExecutor(3) as pool:
        jobs = [pool.submit(pkg.lms.estimate_ir, x, x, 12, 1e-3, 1) for _ in range(4)]
        while not all(j.done() for j in jobs):
            pkg.lms.release()
        assert all(np.array_equal(j.result(), first) for j in jobs)
    # another allocation takes what is kept
    pkg.lms.estimate_ir(x, x, 12, 1e-3, epochs=1)
    assert before - torch.cuda.mem_get_info()[0] > 300 * MB
    block = torch.empty(torch.cuda.mem_get_info()[0] + 200 * MB, dtype=torch.uint8, device="cuda")
    del block
    torch.cuda.empty_cache()
    pkg.lms.release()
    assert before - torch.cuda.mem_get_info()[0] < 40 * MB
    with pytest.raises(pkg.AfdError):
        pkg.lms.release(device=99)
