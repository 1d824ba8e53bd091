"""The REF-mode PML in units of four cells and slab boxes against the CPU
oracle, bit for bit (the same expressions in the same order)."""
import numpy as np
import pytest

import oracle
from test_gpu_parity import run_gpu
from test_gpu_resident import room

pytestmark = pytest.mark.gpu


# ragged rows, one cell a row, slabs that are empty (width 1, 2), reach one
# cell inside (3), meet and overlap (half and all of the grid), two members
@pytest.mark.parametrize("dims,width", [((5, 6, 7), 4), ((31, 18, 22), 1), ((30, 18, 22), 2), ((29, 19, 21), 3),
                                        ((34, 23, 20), 10), ((33, 17, 16), 12), ((21, 20, 19), 30), ((66, 41, 33), 8)])
def test_ref_pml_matches_oracle(pkg, dims, width):
    nx, ny, nz = dims
    vox, a, b = room(nx, ny, nz, 2, width)
    rng = np.random.default_rng(width)
    ksi = [np.concatenate([rng.uniform(0, 6000, min(width, n)), np.zeros(max(n - 2 * width, 0)),
                           rng.uniform(0, 6000, n)])[:n].astype(np.float32) for n in dims]
    sig = rng.standard_normal(60).astype(np.float32)
    srcs, rcv = [((nx // 2, ny // 2, nz // 2), sig)], [(2, 2, 2), (nx - 3, ny - 3, nz - 3), (nx // 2, 3, 3)]
    kw = dict(mode=0, pml=(width, 63, ksi), runs=[70])
    got, field, _ = run_gpu(pkg, dims, vox, a, b, srcs, rcv, 70, **kw)
    want, wfield = oracle.simulate(dims, vox, a, b, mode=0, pml_width=width, faces=63, ksi=ksi, sources=srcs,
                                   receivers=rcv, steps=70, want_field=True)
    assert np.array_equal(got, want) and np.array_equal(field, wfield)
