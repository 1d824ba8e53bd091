"""Which of its routes a run takes (afd_info.resident) and that each gives the
oracle's bits: small grids run all steps of a chunk in the resident kernel; a
capture, a forced plan, launches without graphs and larger grids run the steps as
launches of their own, in replayed graphs whose plan the autotuner chooses.
Everything evaluates the same expressions in the same order: tolerance zero."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import oracle
from test_gpu_resident import room

pytestmark = pytest.mark.gpu


def build(pkg, dims, mode, faces, storage, seed=3, K=3, **params):
    """A walled room, open and absorbing at `faces` (all six: free space around
    one obstacle), four sources and four receivers."""
    W = pkg.workloads
    nx, ny, nz = dims
    vox, a, b = room(nx, ny, nz, K, K)
    if faces & 32:
        vox[-1] = -1
    if faces & 2:
        vox[:, :, -1] = -1
    if faces == 63:
        vox[:] = -1
        vox[nz // 2 - 3:nz // 2 + 3, ny // 2 - 3:ny // 2 + 3, nx // 2 - 3:nx // 2 + 3] = 1
    vox = W.close_gaps(vox)
    ksi = W.ksi_arrays(dims, 8, faces, kmax=6000.0) if faces else None
    rng = np.random.default_rng(seed)
    cells = [(nx // 2, ny // 2, 11), (nx // 2, ny // 2, 11), (12, 11, 11), (nx // 2 + 3, ny // 2, nz // 2)]
    srcs = [(c, (0.5 * rng.standard_normal(180)).astype(np.float32)) for c in cells]
    rcv = [(nx // 2, ny // 2, 12), (11, 11, 11), (nx - 12, ny - 12, nz - 12), (4, 4, 4)]
    sim = pkg.Simulation(mode=mode, storage=storage, dx=0.02, c=340.0, dt=3.125e-5, **params)
    sim.SetModel(pkg.Model.from_voxels(vox, a, b))
    if faces:
        sim.SetPml(8, faces=faces, ksi=ksi)
    for c, s in srcs:
        sim.AddSourceCell(c, s)
    for r in rcv:
        sim.AddMicCell(r)
    args = dict(mode=mode, sources=srcs, receivers=rcv, want_field=True, precision="f16" if storage else "f32")
    if faces:
        args.update(pml_width=8, faces=faces, ksi=ksi)
    return sim, (dims, vox, a, b), args


# the graph order of a single member: streaming kernel, boundary kernel with the
# sources and receivers beside the PML pressure, auxiliary fields; psi kept with
# six faces
@pytest.mark.parametrize("route", ["resident", "capture", "plan", "serial"])
@pytest.mark.parametrize("mode,faces,storage", [(0, 0, 0), (1, 0, 0), (1, 32, 0), (1, 63, 0), (1, 34, 1), (1, 63, 1)])
def test_routes_of_small_rooms_match_the_oracle(pkg, route, mode, faces, storage):
    dims, runs = (48, 45, 43), [1, 203, 40]
    sim, geo, args = build(pkg, dims, mode, faces, storage, graphs=0 if route == "serial" else 1)
    if route == "capture":
        sim.set_capture(2, 20, 50)
    if route == "plan":
        sim.set_plan()
    for n in runs:
        sim.Run(n)
        assert sim.info().resident == (route == "resident")
    want, wfield = oracle.simulate(*geo, runs=runs, **args)
    assert np.array_equal(sim.mics(), want) and np.array_equal(sim.field(), wfield)
    sim.close()


@pytest.mark.parametrize("storage", [0, 1])
def test_tuned_single_room_above_the_resident_size(pkg, storage):
    """One room of 6.6 M cells with an absorbing face, long enough for every
    candidate plan: the tuner ends, and the run equals the serial one."""
    out = []
    for graphs in (1, 0):
        sim, _, _ = build(pkg, (224, 176, 168), 1, 32, storage, graphs=graphs)
        sim.Run(3401)
        tuning = bool(sim.info().tuned)
        sim.Run(199)
        info = sim.info()
        assert not info.resident and tuning == bool(info.tuned) == bool(graphs)
        out.append((sim.mics(), sim.field()))
        sim.close()
    assert np.abs(out[0][0]).max() > 0
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


def test_resident_rooms_on_threads(pkg):
    """Resident kernels of several simulations at a time (each a cooperative
    launch whose blocks wait for one another): the results of each alone."""
    forms = [((48, 45, 43), 1, 63, 0), ((48, 45, 43), 0, 0, 0), ((120, 96, 80), 1, 32, 0), ((120, 96, 80), 1, 34, 1)]

    def run(f):
        sim, _, _ = build(pkg, *f)
        for _ in range(4):
            sim.Run(250)
        assert sim.info().resident == 1
        out = sim.mics(), sim.field()
        sim.close()
        return out

    alone = [run(f) for f in forms]
    with ThreadPoolExecutor(4) as pool:
        beside = list(pool.map(run, forms * 2))
    for k, got in enumerate(beside):
        for a, b in zip(got, alone[k % 4]):
            assert np.array_equal(a, b), forms[k % 4]


@pytest.mark.parametrize("route", ["resident", "capture", "plan"])
@pytest.mark.parametrize("mode,storage", [(0, 0), (1, 0), (1, 1)])
def test_pml_set_again_between_runs(pkg, route, mode, storage):
    """A PML set, set again and taken off between runs starts its fields anew at that
    step on every route: the bits of the serial one."""
    dims, out = (48, 45, 43), []
    W = pkg.workloads
    for r in (route, "serial"):
        sim, _, _ = build(pkg, dims, mode, 0, storage, graphs=0 if r == "serial" else 1)
        if r == "capture":
            sim.set_capture(2, 20, 50)
        if r == "plan":
            sim.set_plan()
        for k, n in enumerate((31, 202, 7, 40)):
            if k:
                width = (0, 8, 8, 0)[k]
                sim.SetPml(width, faces=63 if width else 0, ksi=W.ksi_arrays(dims, 8, 63, kmax=3000.0 * k))
            sim.Run(n)
        out.append((sim.mics(), sim.field()))
        sim.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
