"""The resident kernel, which runs all steps of a chunk for grids that stay in
L2, against the CPU oracle and against the step's separate launches (graphs=0)
bit for bit: both evaluate the same expressions in the same order, so the
tolerance is zero. FP16 with a source on an outer face is compared with the
launches alone: the scales follow the largest inner value, the oracle's the
largest of all (test_gpu_fp16 has the oracle for inner sources, which take the
same kernel)."""
import numpy as np
import pytest

import oracle
from test_gpu_parity import run_gpu

pytestmark = pytest.mark.gpu


def room(nx, ny, nz, K, seed):
    import ancfield_b200.workloads as W
    rng = np.random.default_rng(seed)
    vox = -np.ones((nz, ny, nx), np.int32)
    vox[0], vox[-1], vox[:, 0], vox[:, -1], vox[:, :, 0], vox[:, :, -1] = 0, 1, 2, 0, 1, 2
    if min(nx, ny, nz) > 12:
        vox[5:8, 6:9, 7:11] = 1
    a = (rng.uniform(0.02, 0.5, (3, K)) * np.array([1.0] + [0.3] * (K - 1))).astype(np.float32)
    b = rng.uniform(-0.4, 0.4, (3, K)).astype(np.float32)
    b[:, 0] = 1.0
    return W.close_gaps(vox), a, b


# mode, dims, K, PML faces, storage, steps per run: one unit a row and ragged
# rows, run-time K (5), slabs on no / one / six faces, chunk remainders
@pytest.mark.parametrize("mode,dims,K,faces,storage,runs", [
    (0, (5, 5, 5), 1, 0, 0, [7]), (0, (31, 18, 22), 2, 0, 0, [1, 200, 3]), (0, (66, 33, 21), 5, 0, 0, [201]),
    (1, (37, 40, 35), 3, 0, 0, [205]), (1, (48, 39, 37), 2, 32, 0, [150, 60]), (1, (44, 45, 43), 4, 63, 0, [90]),
    (1, (35, 21, 18), 1, 0, 1, [201]), (1, (48, 39, 37), 5, 34, 1, [130, 75])])
def test_resident_matches_oracle_and_launches(pkg, mode, dims, K, faces, storage, runs):
    import ancfield_b200.workloads as W
    nx, ny, nz = dims
    vox, a, b = room(nx, ny, nz, K, K)
    if faces & 32:
        vox[-1] = -1
    if faces & 2:
        vox[:, :, -1] = -1
    if faces == 63:
        vox[:] = -1
        vox[18:24, 18:25, 17:26] = 1
    vox = W.close_gaps(vox)
    pml = (8, faces, W.ksi_arrays(dims, 8, faces, kmax=6000.0)) if faces else None
    rng = np.random.default_rng(3)
    n = sum(runs)
    # two sources in one air cell, one in a boundary cell, one on an outer face
    cells = [(nx // 2, ny // 2, 2), (nx // 2, ny // 2, 2), (2, 1, 2), (0, 2, 2)]
    srcs = [(c, (0.5 * rng.standard_normal(n - 20 if n > 20 else n)).astype(np.float32)) for c in cells]
    rcv = [(nx // 2, ny // 2, 2), (1, 1, 1), (nx - 2, ny - 2, nz - 2), (0, 2, 2)]
    kw = dict(mode=mode, pml=pml, runs=runs, storage=storage)
    got, field, _ = run_gpu(pkg, dims, vox, a, b, srcs, rcv, n, **kw)
    gen, gfield, _ = run_gpu(pkg, dims, vox, a, b, srcs, rcv, n, graphs=0, **kw)
    assert np.array_equal(got, gen) and np.array_equal(field, gfield)
    if storage:
        return
    args = dict(mode=mode, sources=srcs, receivers=rcv, runs=runs, want_field=True)
    if pml:
        args.update(pml_width=8, faces=faces, ksi=pml[2])
    want, wfield = oracle.simulate(dims, vox, a, b, **args)
    assert np.array_equal(got, want) and np.array_equal(field, wfield)


# members side by side, one of them silent; more source cells than the step's
# kernels take (the separate launches run); a capture switched on and off
# between runs (the route changes within one simulation)
@pytest.mark.parametrize("mode,storage", [(0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("form", ["batch", "many", "switch"])
def test_resident_routes(pkg, mode, storage, form):
    dims = (34, 27, 23)
    vox, a, b = room(*dims, 2, 9)
    rng = np.random.default_rng(5)
    batch = 5 if form == "batch" else 1
    out = []
    for graphs in (1, 0):
        sim = pkg.Simulation(mode=mode, storage=storage, dx=0.02, c=340.0, dt=3.125e-5, batch=batch, graphs=graphs)
        sim.SetModel(pkg.Model.from_voxels(vox, a, b))
        rng = np.random.default_rng(5)
        for k in range(300 if form == "many" else 4):
            cell = (2 + k % 29, 2 + k // 29 % 22, 2 + k // 300)
            sim.AddSourceCell(cell, rng.standard_normal(60).astype(np.float32), batch=k % max(1, batch - 1))
        sim.AddMicCell((20, 12, 11))
        sim.AddMicCell((3, 2, 2))
        for r in range(3):
            if form == "switch":
                sim.set_capture(2, 11, 10 if r == 1 else 0)
            sim.Run(53)
        out.append([np.array([f(b_) for b_ in range(batch)]) for f in (sim.mics, sim.field)])
        sim.close()
    assert np.abs(out[0][0]).max() > 0
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


# the record's spare room (8192 steps) used up exactly, passed by one, and with
# a receiver added on the way; every run against one run of the same length.
# capture: the steps' own launches in graphs that outlive the runs
@pytest.mark.parametrize("capture", [0, 5000])
@pytest.mark.parametrize("runs", [[1, 8192, 1, 200], [100, 8093, 300], [300, 7]])
def test_record_grows_over_runs(pkg, capture, runs):
    dims = (20, 14, 12)
    vox, a, b = room(*dims, 2, 3)
    n = sum(runs)
    sig = np.random.default_rng(8).standard_normal(n).astype(np.float32)
    out = []
    for steps in (runs, [n]):
        sim = pkg.Simulation(mode=1, dx=0.02, c=340.0, dt=3.125e-5)
        sim.SetModel(pkg.Model.from_voxels(vox, a, b))
        sim.AddSourceCell((5, 6, 7), sig)
        sim.AddMicCell((9, 9, 9))
        if capture:
            sim.set_capture(2, 6, capture)
        for k, r in enumerate(steps):
            if k == len(steps) - 1 and len(steps) > 1:
                sim.AddMicCell((3, 2, 2))
            sim.Run(r)
        out.append((np.array(sim.mics()), np.array(sim.field())))
        sim.close()
    (m0, f0), (m1, f1) = out
    assert m0.shape == (2, n) and np.array_equal(m0[0], m1[0]) and np.array_equal(f0, f1)
    assert not m0[1, :n - runs[-1]].any()
