"""The REF-mode PML kernels in their forms, by cells of all members: one cell a
thread (test_gpu_ref_pml has the small grids), units of four with the slabs' rows
spread over more blocks, and whole planes a block; against the CPU oracle, bit for
bit (the same expressions in the same order)."""
import numpy as np
import pytest

import oracle
from test_gpu_resident import room

pytestmark = pytest.mark.gpu


# both sides of the first line (120000 cells); slabs that are empty (width 1, 2),
# reach one cell inside (3), meet and fill the grid; rows that end within a unit;
# members, of which the first and the last have sources; the second line (a million)
@pytest.mark.parametrize("dims,width,batch", [
    ((54, 54, 52), 5, 1), ((55, 55, 52), 5, 1), ((71, 64, 53), 1, 1), ((70, 64, 53), 2, 1), ((69, 64, 53), 3, 1),
    ((72, 61, 53), 9, 1), ((71, 64, 53), 34, 1), ((71, 64, 53), 70, 1), ((21, 20, 19), 4, 40), ((11, 9, 30), 6, 190),
    ((131, 102, 95), 4, 1), ((130, 101, 97), 13, 1), ((28, 22, 18), 5, 180)])
def test_units_of_four_match_oracle(pkg, dims, width, batch):
    nx, ny, nz = dims
    vox, a, b = room(nx, ny, nz, 2, width)
    rng = np.random.default_rng(width)
    ksi = [np.concatenate([rng.uniform(0, 6000, min(width, n)), np.zeros(max(n - 2 * width, 0)),
                           rng.uniform(0, 6000, n)])[:n].astype(np.float32) for n in dims]
    rcv = [(2, 2, 2), (nx - 3, ny - 3, nz - 3), (nx // 2, 3, 3)]
    sigs = {m: rng.standard_normal(40).astype(np.float32) for m in {0, batch - 1}}
    cell = (nx // 2, ny // 2, nz // 2)
    sim = pkg.Simulation(mode=0, dx=0.02, c=340.0, dt=3.125e-5, batch=batch)
    sim.SetModel(pkg.Model.from_voxels(vox, a, b))
    sim.SetPml(width, faces=63, ksi=ksi)
    for m, sig in sigs.items():
        sim.AddSourceCell(cell, sig, batch=m)
    for r in rcv:
        sim.AddMicCell(r)
    sim.Run(45)
    for m in sorted({0, batch // 2, batch - 1}):
        srcs = [(cell, sigs[m])] if m in sigs else []
        want, wfield = oracle.simulate(dims, vox, a, b, mode=0, pml_width=width, faces=63, ksi=ksi, sources=srcs,
                                       receivers=rcv, steps=45, want_field=True)
        assert np.array_equal(sim.mics(m), want) and np.array_equal(sim.field(m), wfield)
    sim.close()


def test_thin_layers_of_many_members_are_not_slower(pkg):
    """64 members of 28x22x18: a layer of 4 cells takes no longer than one of 8 (with
    a block per plane and slab it took a quarter longer), best of several runs."""
    dims = (28, 22, 18)
    vox, a, b = room(*dims, 2, 1)
    ms = {}
    for width in (4, 8):
        sim = pkg.Simulation(mode=0, dx=0.02, c=340.0, dt=3.125e-5, batch=64)
        sim.SetModel(pkg.Model.from_voxels(vox, a, b))
        sim.SetPml(width, faces=63, ksi=pkg.workloads.ksi_arrays(dims, width, 63, kmax=6000.0))
        sim.AddSourceCell((14, 11, 9), np.ones(20, np.float32))
        v = []
        for _ in range(5):
            sim.Run(400)
            v.append(sim.info().last_run_ms)
        ms[width] = min(v[1:])
        sim.close()
    assert ms[4] < 1.1 * ms[8]
