"""Sources and receivers of many members: each member takes its own source cells
and leaves the others' to its ordinary update, on every route that has them in the
step's own kernels, bit for bit as separate source/receiver launches do; and the
resident step is no slower than launches however many there are."""
import numpy as np
import pytest

from test_gpu_resident import room

pytestmark = pytest.mark.gpu


def build(pkg, dims, batch, srcs, rcv, mode=1, storage=0, pml=False, **params):
    W = pkg.workloads
    vox, a, b = room(*dims, 2, 9)
    if pml:
        vox[-1] = -1
        vox = W.close_gaps(vox)
    sim = pkg.Simulation(mode=mode, storage=storage, dx=0.02, c=340.0, dt=3.125e-5, batch=batch, **params)
    sim.SetModel(pkg.Model.from_voxels(vox, a, b))
    if pml:
        sim.SetPml(8, faces=32, ksi=W.ksi_arrays(dims, 8, 32, kmax=6000.0))
    for m, cell, sig in srcs:
        sim.AddSourceCell(cell, sig, batch=m)
    for r in rcv:
        sim.AddMicCell(r)
    return sim


# cells in a wall's boundary layer, on an outer face and inside, of one member, of
# some, of all, twice in one member; a silent member; more pairs than a warp, and
# than a group; one member. Receivers more than a group's threads
@pytest.mark.parametrize("mode,storage,pml", [(0, 0, False), (1, 0, True), (1, 1, False), (1, 1, True)])
@pytest.mark.parametrize("batch,per_member,receivers", [(7, 0, 3), (40, 9, 20), (1, 70, 300), (3, 120, 0)])
def test_own_cells_of_each_member(pkg, mode, storage, pml, batch, per_member, receivers):
    dims = (34, 27, 35)
    nx, ny, nz = dims
    rng = np.random.default_rng(batch)
    srcs = []

    def add(m, cell):
        srcs.append((m, cell, rng.standard_normal(50).astype(np.float32)))

    wall, inside, outer, shared = (1, 9, 12), (15, 12, 10), (0, 9, 12), (16, 12, 10)
    for m in range(batch - 1 if batch > 1 else 1):  # the last of several members is silent
        add(m, shared)
        if m % 3 == 0:
            add(m, wall)
            add(m, wall)
        if m % 3 != 1:
            add(m, inside)
        if m % 4 == 1:
            add(m, outer)
        for k in range(per_member):  # cells that neighbouring members share in part
            q = (per_member // 3 * m + k) % 240
            add(m, (1 + q % 30, 2 + q // 30 * 3, 8 + q % 2))
    rcv = [shared, inside, wall, (30, 20, 20)] + [(1 + k % 32, 1 + k % 25, 1 + k % 33) for k in range(receivers)]
    out = []
    for route in ("resident", "capture", "serial"):
        sim = build(pkg, dims, batch, srcs, rcv, mode, storage, pml, graphs=0 if route == "serial" else 1)
        if route == "capture":
            sim.set_capture(2, 6, 40)
        for n in (3, 60):
            sim.Run(n)
        assert sim.info().resident == (route == "resident")
        out.append([np.array([f(b) for b in range(batch)]) for f in (sim.mics, sim.field)])
        sim.close()
    assert np.abs(out[0][0]).max() > 0
    for other in out[1:]:
        assert np.array_equal(out[0][0], other[0]) and np.array_equal(out[0][1], other[1])


def test_receivers_and_sources_added_between_runs(pkg):
    """Their share of the resident step changes with them."""
    dims = (34, 27, 35)
    out = []
    for graphs in (1, 0):
        sim = build(pkg, dims, 6, [(0, (9, 9, 9), np.ones(30, np.float32))], [(9, 9, 12)], graphs=graphs)
        rng = np.random.default_rng(1)
        for k in range(5):
            sim.Run(21)
            for q in range(300 if k == 1 else 1):
                sim.AddMicCell((2 + q % 30, 3 + k, 4))
            for m in range(k, 6):
                sim.AddSourceCell((4 + 3 * m, 9, 10 + k), rng.standard_normal(80).astype(np.float32), batch=m)
        sim.Run(21)
        out.append(np.array([sim.mics(b) for b in range(6)]))
        sim.close()
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("storage", [0, 1])
@pytest.mark.parametrize("batch,receivers", [(256, 4), (128, 4), (16, 1000), (1, 4000)])
def test_many_are_no_slower_than_launches(pkg, storage, batch, receivers):
    """A source of its own in every member of a 28x22x18 room: best of several
    runs, in turn with a forced plan of the launches."""
    dims = (28, 22, 18)
    sig = np.ones(50, np.float32)
    srcs = [(m, (2 + m % 24, 2 + m // 24 % 18, 3), sig) for m in range(batch)]
    rcv = [(2 + k % 24, 2 + k // 24 % 18, 2 + k // 432 % 14) for k in range(receivers)]
    sims = [build(pkg, dims, batch, srcs, rcv, storage=storage) for _ in range(2)]
    sims[1].set_plan()
    ms = [[], []]
    for _ in range(6):
        for k, sim in enumerate(sims):
            sim.Run(200)
            ms[k].append(sim.info().last_run_ms)
    assert [s.info().resident for s in sims] == [1, 0]
    assert min(ms[0][1:]) < 1.1 * min(ms[1][1:])
    for sim in sims:
        sim.close()


def test_near_the_largest_size_of_the_resident_step(pkg):
    """42 members of 64x48x40, 5.2 M cells with 560000 boundary entries: columns so
    long that whole passes of them left the groups uneven took 1.45 times the launches
    of a fixed plan; the present ones are within a quarter."""
    dims = (64, 48, 40)
    srcs = [(m, (30, 20, 10), np.ones(50, np.float32)) for m in range(42)]
    sims = [build(pkg, dims, 42, srcs, [(12, 12, 12)]) for _ in range(2)]
    sims[1].set_plan()
    ms = [[], []]
    for _ in range(6):
        for k, sim in enumerate(sims):
            sim.Run(300)
            ms[k].append(sim.info().last_run_ms)
    assert [s.info().resident for s in sims] == [1, 0]
    assert min(ms[0][1:]) < 1.25 * min(ms[1][1:])
    assert np.array_equal(sims[0].field(17), sims[1].field(17))
    for sim in sims:
        sim.close()
