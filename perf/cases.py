"""Work that users of the framework have it do, through its public entry points.

Three kinds of case:

fdtd   the acoustic simulation, the framework's main path. `job` cases take a room from its voxels to
       the receivers' signals, as the command line's load/run/save does: a Simulation is made, run and
       closed in each pass. The others keep a Simulation that is running and advance it by `steps` more
       time steps: receivers' new samples and the picture plane (the command line's `vis`) come back.
lms    identification of an impulse response from a recording (EstimateIr).
gemm   the BF16 GEMM under the learned surrogate.
mlp    training steps of the learned surrogate, the weights read at the end.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "ancfield_b200" in sys.modules:
        return sys.modules["ancfield_b200"]
    home = os.path.join(ROOT, "anc-field_b200")
    spec = importlib.util.spec_from_file_location("ancfield_b200", os.path.join(home, "__init__.py"),
                                                  submodule_search_locations=[home])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["ancfield_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


DX, SOUND = 0.025, 343.0
DT = 0.99 / math.sqrt(3.0) * DX / SOUND
TUNING = 1801       # steps of a kept simulation before the first pass (the plan tuner has settled)
SIGNAL = 1 << 17    # source samples of a kept simulation; silence follows


def _fdtd(name, dims, mode, K, steps, storage="fp32", batch=1, pml=0, faces=0, boxes=1, mics=8, signal="noise",
          job=False):
    return {"name": name, "kind": "fdtd", "nx": dims[0], "ny": dims[1], "nz": dims[2], "mode": mode, "K": K,
            "steps": steps, "storage": storage, "batch": batch, "pml": pml, "faces": faces, "boxes": boxes,
            "mics": mics, "signal": signal, "job": job}


def listed():
    return [
        # the smallest rooms users start with (and the framework's known-answer rooms): launches count
        _fdtd("tiny_ref", (28, 22, 18), "ref", 2, 160, boxes=1, mics=4),
        # one impulse response of a living room, from voxels to signals (the C1 room): set-up and run
        _fdtd("c1_job", (160, 120, 100), "fixed", 2, 2000, pml=12, faces=32, signal="pulse", job=True),
        # the same room with the reference's own absorbing layer (whole interior), advanced in parts
        _fdtd("c1_refpml", (160, 120, 100), "ref", 2, 400, pml=12, faces=63),
        # a hall of the shipped ie224 model's size in the command line's default mode (constant admittances)
        _fdtd("hall_ref", (416, 160, 576), "ref", 1, 200, boxes=8, mics=14),
        # free field around obstacles: absorbing layer on all six faces, uneven edges, third-order filters
        _fdtd("sixface_ragged", (204, 157, 131), "fixed", 4, 400, pml=12, faces=63, boxes=6, mics=16),
        # the headline workload: 63 M cells, 20 pieces of furniture, two open faces, 32 receivers
        _fdtd("c2_fp32", (512, 384, 320), "fixed", 4, 400, pml=12, faces=34, boxes=20, mics=32),
        # the same with FP16 field storage
        _fdtd("c2_fp16", (512, 384, 320), "fixed", 4, 400, storage="fp16", pml=12, faces=34, boxes=20, mics=32),
        # 16 secondary paths of one room at once (the C3 batch)
        _fdtd("c3_batch16", (256, 192, 160), "fixed", 2, 200, batch=16, pml=12, faces=32, mics=16, signal="impulse"),
        # identification at the shipped example's filter length (64000 taps), part of its recording and passes
        {"name": "lms_64000", "kind": "lms", "taps": 64000, "samples": 128000, "epochs": 4},
        # the readout's normal equations (the bench's GEMM) and its answer for one block of receiver positions
        {"name": "gemm_fit", "kind": "gemm", "m": 8192, "n": 4096, "k": 4096},
        {"name": "gemm_readout", "kind": "gemm", "m": 128, "n": 2048, "k": 8192},
        # part of an epoch of the surrogate at its default size
        {"name": "mlp_train", "kind": "mlp", "freq": 128, "hidden": 512, "layers": 5, "out": 2048, "batch": 1024,
         "steps": 32},
    ]


def _log(rng, lo, hi, step=1):
    """A whole multiple of `step` in lo .. hi, even in its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + step * 0.999)))
    return int(max(lo, min(hi, v // step * step)))


def draw(rng):
    kind = rng.choices(("fdtd", "lms", "gemm", "mlp"), (8, 2, 2, 1))[0]
    if kind == "lms":
        taps, epochs = _log(rng, 500, 64000), rng.choice((1, 2, 4, 8, 16))
        most = min(320000, 512000 // epochs)
        return {"kind": "lms", "taps": taps, "samples": _log(rng, 4000, most), "epochs": epochs}
    if kind == "gemm":
        m, n, k = _log(rng, 128, 8192, 128), _log(rng, 128, 8192, 128), _log(rng, 64, 8192, 64)
        while m * n * k > 8192 * 4096 * 4096:
            k = max(64, k // 2 // 64 * 64)
        return {"kind": "gemm", "m": m, "n": n, "k": k}
    if kind == "mlp":
        return {"kind": "mlp", "freq": rng.choice((64, 128, 192)), "hidden": 128 * rng.randint(1, 6),
                "layers": rng.randint(3, 6), "out": _log(rng, 128, 2048, 128), "batch": _log(rng, 128, 1024, 128),
                "steps": rng.randint(8, 32)}
    # a room of 20 to 512 cells an edge: its volume even in its logarithm, its proportions within 1 : 3
    cells = math.exp(rng.uniform(math.log(8e3), math.log(60e6)))
    e = [rng.uniform(1.0, 3.0) for _ in range(3)]
    f = (cells / (e[0] * e[1] * e[2])) ** (1.0 / 3.0)
    dims = [max(20, min(576, int(v * f))) for v in e]
    mode = rng.choice(("ref", "fixed", "fixed"))
    storage = "fp16" if mode == "fixed" and rng.random() < 0.3 else "fp32"
    vol = dims[0] * dims[1] * dims[2]
    batch = min(rng.choice((1, 1, 1, 2, 4, 8, 16)), max(1, int(63e6 // vol)))
    pml = rng.choice((0, 8, 12)) if mode == "fixed" else rng.choice((0, 0, 0, 8)) if vol < 4e6 else 0
    pml = pml if min(dims) >= 3 * pml else 0
    faces = (63 if mode == "ref" else rng.choice((1, 2, 8, 16, 32, 34, 48, 63))) if pml else 0
    if faces & 3:  # an absorbing layer along x on rows of whole 4-cell units
        dims[0] -= dims[0] % 4
    c = _fdtd("", dims, mode, rng.randint(1, 4), 200 if vol * batch > 4e6 else 400, storage, batch, pml, faces,
              rng.randint(0, 12), rng.randint(1, 32), rng.choice(("noise", "pulse", "impulse")))
    del c["name"]
    return c


# ---- inputs -----------------------------------------------------------------
def _room(case, rng):
    """int32 voxels [nz, ny, nx] of a room of 3 materials: walls on the faces without an absorbing layer
    (every face in "ref"), boxes as furniture, each in a block of its own so that no gap is one cell wide."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    vox = np.full((nz, ny, nx), -1, np.int32)
    open_ = case["faces"] if case["mode"] == "fixed" and case["pml"] else 0
    mats = rng.integers(0, 3, 6)
    for face, at in enumerate(((Ellipsis, 0), (Ellipsis, -1), (slice(None), 0), (slice(None), -1), 0, -1)):
        if not open_ >> face & 1:
            vox[at] = mats[face]
    lo = max(6, case["pml"] + 4)
    axes = []
    for n in (nx, ny, nz):
        blocks = max(1, min(4, (n - 2 * lo) // 14))
        size = (n - 2 * lo) // blocks
        axes.append([(lo + i * size, size) for i in range(blocks)] if size >= 7 else [])
    places = [(a, b, c) for a in axes[0] for b in axes[1] for c in axes[2]]
    for k in rng.permutation(len(places))[:case["boxes"]]:
        cut = []
        for at, size in places[k]:
            w = int(rng.integers(3, max(4, min(60, size - 4) + 1)))
            s = at + int(rng.integers(0, size - 3 - w + 1))
            cut.append(slice(s, s + w))
        vox[cut[2], cut[1], cut[0]] = rng.integers(0, 3)
    return vox


def _air(vox, n, rng, margin):
    nz, ny, nx = vox.shape
    got = []
    while len(got) < n:
        x, y, z = (int(rng.integers(margin, k - margin)) for k in (nx, ny, nz))
        if vox[z, y, x] == -1 and (x, y, z) not in got:
            got.append((x, y, z))
    return got


def _filters(K, rng):
    """Stable, passive admittance filters of 3 materials: sums of first-order sections."""
    a, b = np.zeros((3, K)), np.zeros((3, K))
    for m in range(3):
        if K == 1:
            a[m, 0], b[m, 0] = rng.uniform(0.05, 0.6), 1.0
            continue
        n = K - 1
        g, al, be = rng.uniform(0.05 / n, 0.6 / n, n), rng.uniform(-0.6, 0.6, n), rng.uniform(-0.6, 0.6, n)
        den, num = np.array([1.0]), np.zeros(K)
        for k in range(n):
            den = np.convolve(den, [1.0, be[k]])
            part = np.array([g[k], g[k] * al[k]])
            for j in range(n):
                if j != k:
                    part = np.convolve(part, [1.0, be[j]])
            num += part
        a[m], b[m] = num, den
    return a.astype(np.float32), b.astype(np.float32)


def _source_signal(case, rng, member):
    kind, n = case["signal"], case["steps"] if case["job"] else SIGNAL
    if kind == "impulse":
        return np.array([rng.uniform(0.5, 1.5)], np.float32)
    if kind == "pulse":
        t = np.arange(n if case["job"] else 2000) * DT - 6e-3
        return (np.exp(-(t / 1.5e-3) ** 2) * np.sin(2 * np.pi * rng.uniform(300, 700) * t)).astype(np.float32)
    x = np.fft.rfft(rng.standard_normal(n))   # 50 to 2000 Hz noise of unit power
    f = np.fft.rfftfreq(n, DT)
    x[(f < 50) | (f > 2000)] = 0
    x = np.fft.irfft(x, n)
    return (x / np.sqrt(np.mean(x * x))).astype(np.float32)


def _ksi(case):
    """Damping per axis: a smooth ramp to 8000 1/s toward the faces with an absorbing layer."""
    w = case["pml"]
    d = (w - np.arange(w)) / float(max(w, 1))
    prof = (8000.0 * (d - np.sin(2 * np.pi * d) / (2 * np.pi))).astype(np.float32)
    out = []
    for ax, n in enumerate((case["nx"], case["ny"], case["nz"])):
        k = np.zeros(n, np.float32)
        if case["faces"] >> (2 * ax) & 1:
            k[:w] = prof
        if case["faces"] >> (2 * ax + 1) & 1:
            k[n - w:] = prof[::-1]
        out.append(k)
    return out


def _fdtd_inputs(case, seed):
    rng = np.random.default_rng([seed, 11])
    vox = _room(case, rng)
    a, b = _filters(case["K"], rng)
    margin = max(3, case["pml"] + 2) if case["pml"] else 3
    spots = _air(vox, case["batch"], rng, margin)
    sources = [(spots[m], _source_signal(case, rng, m)) for m in range(case["batch"])]
    return {"vox": vox, "a": a, "b": b, "sources": sources, "mics": _air(vox, case["mics"], rng, 3), "ksi": _ksi(case)}


def _simulation(case, inp):
    P = _package()
    sim = P.Simulation(mode=P.afd.MODE_REF if case["mode"] == "ref" else P.afd.MODE_FIXED, dx=DX, c=SOUND, dt=DT,
                       storage=P.afd.STORE_FP16 if case["storage"] == "fp16" else P.afd.STORE_FP32,
                       batch=case["batch"])
    sim.SetModel(inp["model"])
    if case["pml"]:
        sim.SetPml(case["pml"], faces=case["faces"], ksi=inp["ksi"])
    for m, (cell, sig) in enumerate(inp["sources"]):
        sim.AddSourceCell(cell, sig, batch=m)
    for cell in inp["mics"]:
        sim.AddMicCell(cell)
    return sim


def _lms_inputs(case, seed):
    """A recorded noise and the same through a decaying response. The level keeps the recursion stable
    (mu x taps x power under 0.07)."""
    rng = np.random.default_rng([seed, 12])
    n, taps = case["samples"], case["taps"]
    x = np.fft.rfft(rng.standard_normal(n))
    f = np.fft.rfftfreq(n, 1.0 / 32000.0)
    x[(f < 50) | (f > 8000)] = 0
    x = np.fft.irfft(x, n)
    x *= 0.1 / np.sqrt(np.mean(x * x))
    h = rng.standard_normal(taps) * np.exp(-np.arange(taps) / (taps / 8.0)) * 0.05
    size = 2 ** int(np.ceil(np.log2(n + taps)))
    d = np.fft.irfft(np.fft.rfft(x, size) * np.fft.rfft(h, size), size)[:n]
    return x, d


def _gemm_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(case["m"], case["k"], generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn(case["n"], case["k"], generator=g, device="cuda").to(torch.bfloat16)
    return a, b


def prepare(case, seed):
    P = _package()
    state = {"case": case, "P": P}
    if case["kind"] == "fdtd":
        inp = _fdtd_inputs(case, seed)
        inp["model"] = P.Model.from_voxels(inp.pop("vox"), inp["a"], inp["b"])
        if case["job"]:
            state["inp"] = inp
        else:
            state["sim"] = _simulation(case, inp)
            state["sim"].Run(TUNING)
    elif case["kind"] == "lms":
        state["x"], state["d"] = _lms_inputs(case, seed)
    elif case["kind"] == "gemm":
        state["a"], state["b"] = _gemm_inputs(case, seed)
        state["c"] = torch.empty(case["m"], case["n"], device="cuda")
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = 4 * case["batch"]
        state["x"] = torch.rand(n, 10, generator=g, device="cuda")
        state["y"] = torch.randn(n, case["out"], generator=g, device="cuda")
        state["y"] *= torch.exp(-torch.arange(case["out"], device="cuda") / (case["out"] / 4.0))
        state["net"] = P.surrogate.Mlp(n_freq=case["freq"], hidden=case["hidden"], n_layers=case["layers"],
                                       n_out=case["out"], batch=case["batch"], seed=seed)
        torch.cuda.synchronize()  # the network works on a stream of its own
    return state


def run(state):
    case, P = state["case"], state["P"]
    if case["kind"] == "fdtd":
        sim = _simulation(case, state["inp"]) if case["job"] else state["sim"]
        sim.Run(case["steps"])
        t1 = sim.info().steps_done
        out = {"mics": np.stack([sim.mics_range(t1 - case["steps"], t1, batch=m) for m in range(case["batch"])]),
               "plane": sim.plane(1, case["ny"] // 2)}
        if case["job"]:
            sim.close()
        return out
    if case["kind"] == "lms":
        return P.lms.estimate_ir(state["x"], state["d"], case["taps"], 1e-4, epochs=case["epochs"])
    if case["kind"] == "gemm":
        return P.surrogate.gemm_bf16(state["a"], state["b"], state["c"], torch.cuda.current_stream().cuda_stream)
    net, n = state["net"], case["batch"]
    for i in range(case["steps"]):
        at = i % 4 * n
        last = i == case["steps"] - 1
        loss = net.train_step(state["x"][at:at + n], state["y"][at:at + n], want_loss=last)
    return {"loss": loss, "weights": net.weights()}


# ---- what a pass cannot do without --------------------------------------------
def _surface(case):
    """About the cells beside a wall (the boxes' share depends on the seed and is left out)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    open_ = case["faces"] if case["mode"] == "fixed" and case["pml"] else 0
    face = (ny * nz, ny * nz, nx * nz, nx * nz, nx * ny, nx * ny)
    return sum(f for k, f in enumerate(face) if not open_ >> k & 1)


def _layer(case):
    """Cells of the absorbing layer."""
    if not case["pml"]:
        return 0
    dims, w = (case["nx"], case["ny"], case["nz"]), case["pml"]
    if case["mode"] == "ref":
        return (dims[0] - 4) * (dims[1] - 4) * (dims[2] - 4)
    inner = 1
    for ax, n in enumerate(dims):
        inner *= n - 4 - (w - 2) * ((case["faces"] >> (2 * ax) & 1) + (case["faces"] >> (2 * ax + 1) & 1))
    return (dims[0] - 4) * (dims[1] - 4) * (dims[2] - 4) - inner


def work(case):
    """fdtd: per step two levels read and one written, per wall cell its list entry and filter state, per
    absorbing cell the fields of the layer. lms: per sample taps products for the output and for the update.
    gemm: operands and result once. mlp: per step the weights, their gradients and moments, x and y."""
    if case["kind"] == "fdtd":
        es = 2 if case["storage"] == "fp16" else 4
        inner = (case["nx"] - 2) * (case["ny"] - 2) * (case["nz"] - 2)
        per = 3 * es * inner + _surface(case) * (12 + 8 * case["K"]) + 32 * _layer(case)
        flops = 9 * inner + _surface(case) * (20 + 6 * case["K"]) + 90 * _layer(case)
        return {"bytes": per * case["batch"] * case["steps"], "flops": flops * case["batch"] * case["steps"]}
    if case["kind"] == "lms":
        return {"bytes": 8 * (2 * case["samples"] + case["taps"]),
                "flops": 4 * case["taps"] * case["samples"] * case["epochs"]}
    if case["kind"] == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * k * (m + n) + 4 * m * n, "flops": 2 * m * n * k}
    h, f = case["hidden"], 2 * case["freq"]
    weights = f * h + (case["layers"] - 2) * h * h + h * case["out"]
    return {"bytes": case["steps"] * (32 * weights + 4 * case["batch"] * (10 + case["out"])),
            "flops": case["steps"] * 6 * case["batch"] * weights}


# ---- the same in 64 bits --------------------------------------------------------
_WALLS = [1, 2, 4, 8, 16, 32, 5, 9, 17, 33, 6, 10, 18, 34, 20, 36, 24, 40, 21, 37, 25, 41, 22, 38, 26, 42]


def _exact_fdtd(case, seed):
    inp = _fdtd_inputs(case, seed)
    ref, K, dev, f8 = case["mode"] == "ref", case["K"], "cuda", torch.float64
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    sy, sz, vol = nx, nx * ny, nx * ny * nz
    lam = float(np.float32(DT)) * float(np.float32(SOUND)) / float(np.float32(DX))
    lam2 = lam * lam
    l = lam2 if ref else lam
    l2 = l * l
    c2 = 2 * (1 - 3 * l2)

    def shift(t, d):  # values of the neighbours at distance d, on the flat grid
        return torch.roll(t, -d)

    vox = torch.from_numpy(inp["vox"]).reshape(-1).to(dev)
    solid = vox != -1
    idx = torch.arange(vol, device=dev)
    X, Y, Z = idx % nx, idx // sy % ny, idx // sz
    inner = (X > 0) & (X < nx - 1) & (Y > 0) & (Y < ny - 1) & (Z > 0) & (Z < nz - 1)
    offs = (1, -1, sy, -sy, sz, -sz)
    walls = sum(shift(solid, o).to(torch.int64) << k for k, o in enumerate(offs))
    cell = torch.nonzero(inner & ~solid & (walls > 0)).reshape(-1)
    mask = walls[cell]
    is_wall_cell = torch.zeros(vol, dtype=torch.bool, device=dev)
    is_wall_cell[cell] = True
    # one entry per wall cell: up to three filters in the order of the directions
    nf = sum(mask >> k & 1 for k in range(6))
    mats = torch.zeros(len(cell), 3, dtype=torch.int64, device=dev)
    at = torch.zeros(len(cell), dtype=torch.int64, device=dev)
    for k, o in enumerate(offs):
        has = (mask >> k & 1) == 1
        w = torch.nonzero(has).reshape(-1)
        mats[w, at[w]] = vox[cell[w] + o].to(torch.int64)
        at[w] += 1
    A, B = (torch.from_numpy(inp[k]).double().to(dev) for k in ("a", "b"))
    used = torch.stack([nf > f for f in range(3)], 1)
    width = torch.where((nf == 3) & ref, torch.tensor(K // 2, device=dev), torch.tensor(K, device=dev))
    a0 = torch.where(used, A[mats, 0], 1.0)
    b0 = torch.where(used, B[mats, 0], 1.0)
    kept = (mask == 42) & ref            # the corner that the reference leaves at its interior value
    third = (nf == 3) & ref              # whose third filter does not enter the pressure
    take = torch.where(third[:, None] & (torch.arange(3, device=dev) == 2), torch.zeros((), device=dev, dtype=f8),
                       used.to(f8))
    slots = width[:, None] * torch.arange(3, device=dev)
    dims = (nx, ny, nz)
    W, faces = case["pml"], case["faces"]
    ksi = [torch.from_numpy(np.concatenate([k, np.zeros(max(dims) + 8 - len(k), np.float32)])).double().to(dev)
           for k in inp["ksi"]]
    dt, dx, c = (float(np.float32(v)) for v in (DT, DX, SOUND))
    if W:
        pos = (X, Y, Z)
        slab = [((pos[a] < W) & bool(ref or faces >> (2 * a) & 1)) |
                ((pos[a] > dims[a] - W - 1) & bool(ref or faces >> (2 * a + 1) & 1)) for a in range(3)]
        core = (X > 1) & (X < nx - 2) & (Y > 1) & (Y < ny - 2) & (Z > 1) & (Z < nz - 2)
        pml = core if ref else core & ~solid & ~is_wall_cell & (slab[0] | slab[1] | slab[2])
        pc_ = torch.nonzero(pml).reshape(-1)
        aux = [torch.nonzero(pml & s).reshape(-1) for s in slab]
        kx, ky, kz = (ksi[a][pos[a][pc_]] for a in range(3))
    out = np.zeros((case["batch"], case["mics"], case["steps"]))
    lead = 0 if case["job"] else TUNING
    plane = None
    for member in range(case["batch"]):
        (sx, syy, szz), sig = inp["sources"][member]
        src = szz * sz + syy * sy + sx
        mic = torch.tensor([z * sz + y * sy + x for x, y, z in inp["mics"]], device=dev)
        old, cur = (torch.zeros(vol, dtype=f8, device=dev) for _ in range(2))
        ring = [torch.zeros(len(cell), 3 * K + 1, dtype=f8, device=dev) for _ in range(2)]
        fi = [[torch.zeros(vol, dtype=f8, device=dev) for _ in range(2)] for _ in range(3)] if W else None
        psi = [torch.zeros(vol, dtype=f8, device=dev) for _ in range(2)] if W else None
        row = torch.arange(len(cell), device=dev)[:, None].expand(-1, 3)
        for g in range(lead + case["steps"]):
            new = lam2 * sum(shift(cur, o) for o in offs) + 2 * (1 - 3 * lam2) * cur - old
            new = torch.where(inner, new, old * 0)
            if len(cell):
                ix = K - 1 - g % K
                gn = torch.zeros(len(cell), 3, dtype=f8, device=dev)
                for i in range(1, K):
                    s = torch.where(width[:, None] > 0, (ix + i) % width.clamp(min=1)[:, None], 0) + slots
                    gn += (B[mats, i] * ring[0].gather(1, s) - A[mats, i] * ring[1].gather(1, s)) * used
                S = torch.zeros(len(cell), dtype=f8, device=dev)
                for ax in range(3):
                    up, dn = cur[cell + offs[2 * ax]], cur[cell + offs[2 * ax + 1]]
                    S += torch.where((mask >> (2 * ax) & 1) == 1, 2 * dn,
                                     torch.where((mask >> (2 * ax + 1) & 1) == 1, 2 * up, up + dn))
                y = (l * a0 / b0 * take).sum(1)
                p = (l2 * S + l2 * (gn / b0 * take).sum(1) + c2 * cur[cell] + (y - 1) * old[cell]) / (1 + y)
                p = torch.where(kept, new[cell], p)
                xn = a0 / (l * b0) * (p - old[cell])[:, None] - gn / b0
                yn = (b0 * xn + gn) / a0
                for f in range(3):  # unused filters write the spare slot
                    s = torch.where(used[:, f], ix + slots[:, f], 3 * K)[:, None]
                    ring[0].scatter_(1, s, xn[:, f:f + 1])
                    ring[1].scatter_(1, s, yn[:, f:f + 1])
                new[cell] = p
            if W:
                lv = (g + 1) & 1
                F1 = [fi[a][lv ^ 1] for a in range(3)]
                pm = psi[lv ^ 1][pc_]
                ps = dt * cur[pc_] + pm
                if not ref and faces & 3 and faces & 12 and faces & 48:
                    pass  # psi is kept
                elif not ref:
                    ps, pm = ps * 0, pm * 0

                def avg(t, ax, at):
                    u, v = [o for k, o in enumerate((1, sy, sz)) if k != ax]
                    return 0.25 * (t[at] + t[at + u] + t[at + v] + t[at + u + v])

                def diff(t, ax, at):
                    return avg(t, ax, at + (1, sy, sz)[ax]) - avg(t, ax, at)

                Am = c * c / (dx * dx) * (sum(cur[pc_ + o] for o in offs) - 6 * cur[pc_])
                Bm = sum(diff(F1[a], a, pc_) for a in range(3)) / dx
                ks = (kx + ky + kz) / (2 * dt)
                num = (Am + Bm - kx * ky * kz * 0.5 * (ps + pm) - (old[pc_] - 2 * cur[pc_]) / (dt * dt)
                       - (kx * ky + ky * kz + kz * kx) * cur[pc_] + ks * old[pc_])
                pv = num / (1 / (dt * dt) + ks)
                own_p, own_s = torch.zeros_like(cur), torch.zeros_like(cur)
                if ref:  # a cell's own new values count in its own averages, the others' old ones
                    own_p[pc_], own_s[pc_] = pv - new[pc_], ps - psi[lv][pc_]
                else:
                    new[pc_] = pv
                    psi[lv][pc_] = ps
                for ax in range(3):
                    q = aux[ax]
                    k3 = [0.5 * (ksi[a][pos[a][q]] + ksi[a][pos[a][q] + 1]) for a in range(3)]
                    own = 0.25 * own_p[q]
                    dp = (diff(new, ax, q) - own + avg(cur, ax, q + (1, sy, sz)[ax]) -
                          (avg(new, ax, q) + own if ref else avg(cur, ax, q))) * 0.5 / dx
                    ds = (diff(psi[lv], ax, q) - 0.25 * own_s[q]) / dx
                    o1, o2 = [a for a in range(3) if a != ax]
                    kk = k3[o1] * k3[o2]
                    if ref and ax == 1:
                        kk = 0.5 * (ksi[0][Y[q]] + ksi[0][Y[q] + 1]) * k3[2]
                    f1 = F1[ax][q]
                    fi[ax][lv][q] = ((-0.5 * k3[ax] * f1 + (k3[o1] + k3[o2] - k3[ax]) * dp + kk * ds + f1 / dt) /
                                     (1 / dt + 0.5 * k3[ax]))
                if ref:
                    new[pc_] = pv
                    psi[lv][pc_] = ps
            if g < len(sig):
                new[src] += float(sig[g])
            if g >= lead:
                out[member, :, g - lead] = new[mic].cpu().numpy()
            at_ = g if g < lead or not lead else g - lead  # step of its run
            if W and ref and at_ in (0, 8000):
                for t in (*fi[0], *fi[1], *fi[2], *psi):
                    t.zero_()
            old, cur = cur, new
        if member == 0:
            plane = cur.reshape(nz, ny, nx)[:, ny // 2].cpu().numpy()
    return {"mics": out, "plane": plane}


def _exact_lms(case, seed):
    x, d = _lms_inputs(case, seed)
    n = case["taps"]
    w = np.zeros(n)
    back = np.concatenate([x[::-1], np.zeros(n)])  # back[i:i+n] is the delay line when sample samples-1-i has come
    for _ in range(case["epochs"]):
        for k in range(case["samples"]):
            u = back[case["samples"] - 1 - k:][:n]
            e = d[k] - w @ u
            w += (2 * 1e-4 * e) * u
    return w


def exact(case, seed):
    """None for the training steps (the network's Fourier matrix is drawn inside the library) and where the
    plain form would take too long."""
    if case["kind"] == "gemm":
        a, b = _gemm_inputs(case, seed)
        return a.double() @ b.double().T
    if case["kind"] == "lms" and case["samples"] * case["epochs"] * (4e-6 + case["taps"] * 1.2e-9) < 10:
        return _exact_lms(case, seed)
    if case["kind"] == "fdtd":
        cells = case["nx"] * case["ny"] * case["nz"]
        steps = case["batch"] * (case["steps"] + (0 if case["job"] else TUNING))
        if steps * (2e-3 + cells * (4e-10 + (6e-10 if case["pml"] else 0))) < 15:
            return _exact_fdtd(case, seed)
    return None
