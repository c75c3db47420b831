"""Performance cases: the reconstructions a user of this engine runs, through its public
entry points (`backprojector_gb300.capi`, `backprojector_gb300.octree`).

A case is a dict of plain values.  `prepare` makes what a program has in hand before the
call (captures on the GPU, plans), `run` is one pass, `work` its compulsory bytes and
operations, `exact` the same outputs in FP64 from plain torch.

Captures are made here with torch from the seed: relay wall y = 0, grids over x and z, the
laser and SPAD origins of the engine's synthetic configurations, surface points of a few
hidden spheres behind the wall, each arriving as a short pulse (the detector's timing
jitter, 1.5 bins) with the two legs' fall-off, photon counts with Poisson noise where the
configuration has it.  The learned octree gets scenes from the engine's own renderer, the
distribution its network was trained on.
"""
import math

import numpy as np
import torch

from backprojector_gb300 import capi, octree, synthetic

DEV = "cuda:0"
LASER = (0.0, -0.5, -0.4)
SPAD = (0.0, -0.5, 0.4)
JITTER = 1.5  # bins
UPDATE_FLOPS = 10  # one leg (3 differences, 3 squares summed, root), 2 sums, 1 accumulation
MAX_DRAWN = 3e10   # voxel-pair updates of a drawn case


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # A first look at a coarse scan: the smallest call, a few launches long.
        dict(name="preview_16", kind="dense", scan="single", gx=32, gy=32, T=512, nx=16, ny=16,
             nz=16, wall=1.0, edge=0.5, depth=0.6, rows="f32", kahan=False),
        # The precision configuration: one laser point, 64 x 64 SPADs, 64^3 over 1 m^3.
        dict(name="single_64", kind="dense", scan="single", gx=64, gy=64, T=2048, nx=64, ny=64,
             nz=64, wall=2.0, edge=1.0, depth=1.0, rows="f32", kahan=False),
        # The largest reconstruction: 128 x 128 SPADs, 4096 bins, 256^3 over 1.5 m^3.
        dict(name="single_256", kind="dense", scan="single", gx=128, gy=128, T=4096, nx=256,
             ny=256, nz=256, wall=2.0, edge=1.5, depth=1.0, rows="f32", kahan=False),
        # Exhaustive captures: 16 x 16 lasers x 16 x 16 SPADs.
        dict(name="exhaustive_16", kind="dense", scan="exhaustive", gx=16, gy=16, T=512, nx=32,
             ny=32, nz=32, wall=1.0, edge=0.5, depth=0.6, rows="f32", kahan=False),
        # A confocal raster of no round size into a box of no round size.
        dict(name="confocal_ragged", kind="dense", scan="confocal", gx=61, gy=67, T=1501, nx=90,
             ny=75, nz=101, wall=2.0, edge=1.0, depth=0.9, rows="f32", kahan=False),
        # Laser and SPAD scanned together a fixed distance apart: the pairs do not factor,
        # and the default algorithm choice evaluates the reference's own expression.
        dict(name="offset_scan", kind="dense", scan="offset", gx=64, gy=64, T=2048, nx=64, ny=64,
             nz=64, wall=2.0, edge=1.0, depth=1.0, rows="f32", kahan=False),
        # Phasor field of the phasor configuration: pulse convolution, complex64 rows, 128^3.
        dict(name="phasor_128", kind="phasor", gx=128, gy=128, T=4096, nx=128, ny=128, nz=128,
             wall=2.0, edge=1.5, depth=1.0, rows="c64"),
        # The same with the rows stored as FP16 (re, im) pairs, ragged and smaller.
        dict(name="phasor_half", kind="phasor", gx=50, gy=46, T=1500, nx=61, ny=50, nz=70,
             wall=2.0, edge=1.2, depth=1.0, rows="c32"),
        # The learned octree at its own resolution.
        dict(name="octree_256", kind="octree", gx=128, gy=128, T=4096, n=256, objects=3),
        # Uneven captures in one batch (FP16 rows, graph replays), a quarter of them exhaustive.
        dict(name="batch_24", kind="batch", captures=24, seed=0, exhaustive=0.25),
        # One training step of the occupancy network.
        dict(name="train_16", kind="train", batch=16),
        # The drop-in call on host buffers, a new capture of a known geometry each time.
        dict(name="host_64", kind="host", scan="single", gx=64, gy=64, T=2048, nx=64, ny=64, nz=64,
             wall=2.0, edge=1.0, depth=1.0, rows="f32", kahan=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["dense", "phasor", "host", "octree", "batch", "train"],
                       [14, 4, 2, 2, 2, 1])[0]
    if kind == "octree":
        g = _log_int(rng, 24, 128)
        return dict(kind="octree", gx=g, gy=_log_int(rng, 24, 128), T=4 * _log_int(rng, 256, 1024),
                    n=8 * _log_int(rng, 8, 32), objects=rng.randint(1, 5))
    if kind == "batch":
        return dict(kind="batch", captures=rng.randint(3, 24), seed=rng.randint(1, 10 ** 6),
                    exhaustive=rng.choice([0.0, 0.25, 0.5]))
    if kind == "train":
        return dict(kind="train", batch=rng.randint(2, 16))
    c = dict(kind=kind, gx=_log_int(rng, 12, 128), gy=_log_int(rng, 12, 128),
             T=_log_int(rng, 256, 4096), nx=_log_int(rng, 8, 160), ny=_log_int(rng, 8, 160),
             nz=_log_int(rng, 8, 160), wall=rng.choice([1.0, 2.0]),
             edge=rng.uniform(0.5, 1.5), depth=rng.uniform(0.9, 1.2))
    if kind == "phasor":
        c["rows"] = rng.choice(["c64", "c64", "c32"])
    else:
        c["scan"] = rng.choices(["single", "confocal", "exhaustive", "offset"], [5, 3, 3, 2])[0]
        c["rows"], c["kahan"] = "f32", False
        if c["scan"] == "exhaustive":
            c["gx"], c["gy"] = _log_int(rng, 4, 20), _log_int(rng, 4, 20)
            c["T"] = _log_int(rng, 256, 2048)
        elif c["scan"] != "offset":
            c["rows"], c["kahan"] = rng.choices([("f32", False), ("f16", False), ("bf16", True)],
                                                [5, 3, 2])[0]
    while _updates(c) > MAX_DRAWN:
        for k in ("nx", "ny", "nz"):
            c[k] = max(8, c[k] * 4 // 5)
    return c


# ---------------------------------------------------------------- captures

def _pairs_count(c):
    return (c["gx"] * c["gy"]) ** (2 if c.get("scan") == "exhaustive" else 1)


def _updates(c):
    return float(_pairs_count(c)) * c["nx"] * c["ny"] * c["nz"]


def _grid(nx, nz, size, shift=0.0):
    g = np.zeros((nx, nz, 3), np.float32)
    g[:, :, 0] = np.linspace(-size / 2, size / 2, nx)[:, None] + shift
    g[:, :, 2] = np.linspace(-size / 2, size / 2, nz)[None, :]
    return g.reshape(-1, 3)


def _legs(o, pts):
    d = (np.asarray(o, np.float32) - pts).astype(np.float64)
    return np.sqrt((d * d).sum(1)).astype(np.float32)


def _geometry(c):
    """Pairs, volume basis, t0 and deltaT: the window [t0, t0 + T deltaT) holds every path."""
    scan = c.get("scan", "single")
    spads = _grid(c["gx"], c["gy"], c["wall"])
    if scan == "confocal":
        lasers, cams, lw = spads, spads, _legs(SPAD, spads)
        cw = lw
    elif scan == "offset":
        lasers, cams = _grid(c["gx"], c["gy"], c["wall"], 0.05), spads
        lw, cw = _legs(LASER, lasers), _legs(SPAD, cams)
    else:
        las = spads if scan == "exhaustive" else np.zeros((1, 3), np.float32)
        lasers, lw = np.repeat(las, len(spads), 0), np.repeat(_legs(LASER, las), len(spads))
        cams, cw = np.tile(spads, (len(las), 1)), np.tile(_legs(SPAD, spads), len(las))
    pairs = np.zeros(len(cams), capi.PAIR_DTYPE)
    pairs["laser_point"], pairs["camera_point"] = lasers, cams
    pairs["laser_wall"], pairs["camera_wall"] = lw, cw
    n = np.array([c["nx"], c["ny"], c["nz"]], np.float64)
    pos, size = np.array([0.0, c["depth"], 0.0]), np.full(3, c["edge"])
    lo, hi = pos - size / 2, pos + size / 2
    inc = np.diag(size / (n - 1)).astype(np.float32).reshape(-1)
    near = _box(lasers, lo, hi, False) + _box(cams, lo, hi, False) + lw + cw
    far = _box(lasers, lo, hi, True) + _box(cams, lo, hi, True) + lw + cw
    dt = float(np.float32((far.max() - near.min()) * 1.02 / c["T"]))
    t0 = float(np.float32(math.floor(near.min() / dt) * dt))
    return dict(pairs=pairs, T=c["T"], n=(c["nx"], c["ny"], c["nz"]), zero=lo.astype(np.float32),
                inc=inc, t0=t0, dt=dt, lo=lo, hi=hi)


def _box(p, lo, hi, farthest):
    p = p.astype(np.float64)
    q = np.where(np.abs(p - lo) > np.abs(p - hi), lo, hi) if farthest else np.clip(p, lo, hi)
    return np.sqrt(((p - q) ** 2).sum(1))


def _fields(pairs):
    f = torch.from_numpy(np.ascontiguousarray(pairs).view(np.float32).reshape(-1, 8)).to(DEV)
    return f[:, 0:3], f[:, 3:6], f[:, 6], f[:, 7]  # camera, laser points, camera, laser legs


def _transients(g, seed, peak=1e4, points=48):
    """FP32 rows [P, T] of surface points on three hidden spheres."""
    rng = np.random.default_rng(seed)
    edge = float((g["hi"] - g["lo"]).min())
    pts, alb = [], []
    for _ in range(3):
        r = rng.uniform(0.08, 0.2) * edge
        u = rng.normal(size=(points // 3, 3))
        pts.append(rng.uniform(g["lo"] + r, g["hi"] - r) +
                   r * u / np.linalg.norm(u, axis=1, keepdims=True))
        alb.append(np.full(points // 3, rng.uniform(0.3, 1.0)))
    pts, alb = np.concatenate(pts).astype(np.float32), np.concatenate(alb)
    cam, las, cw, lw = _fields(g["pairs"])
    t = torch.arange(g["T"], device=DEV, dtype=torch.float32)
    H = torch.zeros((len(cw), g["T"]), device=DEV)
    for x, a in zip(torch.from_numpy(pts).to(DEV), alb):
        r1, r2 = (las - x).norm(dim=1), (cam - x).norm(dim=1)
        at = (r1 + r2 + cw + lw - g["t0"]) / g["dt"]
        amp = float(a) / (r1 * r2).square()
        H += torch.exp((t[None, :] - at[:, None]).square_().mul_(-0.5 / JITTER ** 2)) * amp[:, None]
    if peak:
        H *= peak / H.max()
        gen = torch.Generator(device=DEV)
        gen.manual_seed(seed)
        H = torch.poisson(H, generator=gen)
    return H


def _wavelength(c):
    return float(np.float32(4.0 * c["wall"] / (max(c["gx"], c["gy"]) - 1)))


def _pitch(T, esz):
    k = 16 // esz
    return (T + k - 1) // k * k


def _padded(H, pitch):
    if pitch == H.shape[1]:
        return H
    out = torch.zeros((H.shape[0], pitch), device=DEV)
    out[:, :H.shape[1]] = H
    return out


# ---------------------------------------------------------------- dense reconstructions

ROWS = {"f32": (capi.DTYPE_F32, 4), "f16": (capi.DTYPE_F16, 2), "bf16": (capi.DTYPE_BF16, 2)}
TARGET = 16384.0  # half-precision rows: the capture's largest value maps here


def _prepare_dense(c, seed):
    g = _geometry(c)
    dtype, esz = ROWS[c["rows"]]
    pitch = _pitch(c["T"], esz)
    s = dict(kind="dense", P=len(g["pairs"]), T=c["T"], pitch=pitch, dtype=dtype,
             half=c["rows"] != "f32")
    H = _transients(g, seed)
    s["H"] = H if s["half"] else _padded(H, pitch)
    if s["half"]:
        s["rows"] = torch.empty((s["P"], pitch), dtype=torch.int16, device=DEV)
        s["absmax"] = torch.empty(1, device=DEV)
    s["volume"] = torch.empty(g["n"], device=DEV)
    s["plan"] = capi.Plan(g["pairs"], c["T"], g["n"], g["zero"], g["inc"], g["t0"], g["dt"],
                          h_dtype=dtype, h_pitch=pitch,
                          accum=capi.ACCUM_KAHAN if c["kahan"] else capi.ACCUM_F32)
    return s


def _run_dense(s):
    rows = s["H"]
    if s["half"]:
        capi.rows_absmax(s["H"], s["P"], s["T"], s["T"], s["absmax"])
        capi.rows_to_half(s["H"], s["P"], s["T"], s["T"], s["dtype"], s["rows"], s["pitch"],
                          d_absmax=s["absmax"], target=TARGET)
        rows = s["rows"]
    s["plan"].execute(rows, s["volume"])
    if s["half"]:
        capi.volume_scale(s["volume"], s["volume"].numel(), d_absmax=s["absmax"], target=TARGET)
    return s["volume"]


def _prepare_host(c, seed):
    g = _geometry(c)
    return dict(kind="host", g=g, H=_transients(g, seed).cpu().numpy())


def _run_host(s):
    g = s["g"]
    return capi.backproject_host(s["H"], g["pairs"], g["n"], g["zero"], g["inc"], g["t0"], g["dt"])


# ---------------------------------------------------------------- phasor fields

def _prepare_phasor(c, seed):
    g = _geometry(c)
    P, T = len(g["pairs"]), c["T"]
    half = c["rows"] == "c32"
    pitch = _pitch(T, 4)
    s = dict(kind="phasor", P=P, T=T, pitch=pitch, half=half, wavelength=_wavelength(c),
             dt=g["dt"], H=_padded(_transients(g, seed, peak=None), pitch))
    s["field"] = torch.empty((P, pitch), dtype=torch.complex64, device=DEV)
    s["volume"] = torch.empty(g["n"], dtype=torch.complex64, device=DEV)
    if half:
        s["rows"] = torch.empty((P, 2 * pitch), dtype=torch.int16, device=DEV)
        s["absmax"] = torch.empty(1, device=DEV)
    s["plan"] = capi.Plan(g["pairs"], T, g["n"], g["zero"], g["inc"], g["t0"], g["dt"],
                          h_dtype=capi.DTYPE_C32 if half else capi.DTYPE_C64, h_pitch=pitch)
    return s


def _run_phasor(s):
    P, T, pitch = s["P"], s["T"], s["pitch"]
    capi.phasor_pulse_device(s["H"], P, T, pitch, s["wavelength"], s["dt"], s["field"], pitch)
    rows = s["field"]
    if s["half"]:
        capi.rows_absmax(s["field"], P, 2 * T, 2 * pitch, s["absmax"])
        capi.rows_to_half(s["field"], P, 2 * T, 2 * pitch, capi.DTYPE_F16, s["rows"], 2 * pitch,
                          d_absmax=s["absmax"], target=TARGET)
        rows = s["rows"]
    s["plan"].execute(rows, s["volume"])
    if s["half"]:
        capi.volume_scale(s["volume"], 2 * s["volume"].numel(), d_absmax=s["absmax"],
                          target=TARGET)
    return s["volume"]


# ---------------------------------------------------------------- learned octree

def _octree_geometry(c):
    g = _geometry(dict(c, nx=c["n"], ny=c["n"], nz=c["n"], wall=2.0, edge=1.5, depth=1.0))
    return g


def _prepare_octree(c, seed):
    g = _octree_geometry(c)
    P = len(g["pairs"])
    rng = np.random.default_rng(seed)
    spec = synthetic.CaptureSpec("scene", None, (c["gx"], c["gy"]), 2.0, c["T"], g["dt"],
                                 (0.0, 1.0, 0.0), 1.5, c["n"], "objects",
                                 {"count": (c["objects"], c["objects"]),
                                  "kinds": ("sphere", "box", "torus"), "points": 10000,
                                  "albedo": (0.3, 1.0)})
    pts, alb = synthetic.make_scene(spec, rng, g["lo"], g["hi"])
    H = torch.empty((P, c["T"]), device=DEV)
    d_pairs = torch.from_numpy(g["pairs"].view(np.uint8).copy()).to(DEV)
    d_pts, d_alb = torch.from_numpy(pts).to(DEV), torch.from_numpy(alb).to(DEV)
    capi.synth_render_device(d_pairs, P, c["T"], g["t0"], g["dt"], d_pts, d_alb, len(pts), H)
    return dict(kind="octree", H=H, volume=torch.empty(g["n"], device=DEV),
                octree=capi.NativeOctree(g["pairs"], c["T"], g["n"], g["zero"], g["inc"], g["t0"],
                                         g["dt"], octree.WEIGHTS, h_dtype=capi.DTYPE_F16))


def _run_octree(s):
    s["octree"].reconstruct(s["H"], s["volume"])
    return s["volume"]


# ---------------------------------------------------------------- batches

def _batch_captures(c):
    rng = np.random.default_rng(c["seed"])
    out = []
    for _ in range(c["captures"]):
        ex = rng.random() < c["exhaustive"]
        g = 16 if ex else int(rng.choice([16, 32, 48, 64, 96]))
        T = int(rng.choice([512, 1024, 2048]))
        v = int(rng.choice([32, 48, 64, 96]))
        out.append(dict(scan="exhaustive" if ex else "single", gx=g, gy=g, T=T, nx=v, ny=v, nz=v,
                        wall=1.0, edge=0.5, depth=0.6))
    return out


def _batch_parts(c):
    caps = _batch_captures(c)
    geos = [_geometry(k) for k in caps]
    return caps, geos


def _prepare_batch(c, seed):
    caps, geos = _batch_parts(c)
    rows = [_transients(g, seed * 1000 + i, points=12) for i, g in enumerate(geos)]
    scales = [float(H.max()) / TARGET for H in rows]
    batch = capi.Batch([dict(pairs=g["pairs"], T=g["T"], voxels_per_side=g["n"], zero=g["zero"],
                             inc=g["inc"], t0=g["t0"], deltaT=g["dt"], h_scale=k)
                        for g, k in zip(geos, scales)], h_dtype=capi.DTYPE_F16)
    info = batch.info()
    H = torch.zeros((info["total_rows"], info["pitch"]), dtype=torch.float16, device=DEV)
    for r, x, k in zip(batch.row_offsets, rows, scales):
        H[r:r + x.shape[0], :x.shape[1]] = x / k
    return dict(kind="batch", H=H, volumes=torch.empty(info["total_voxels"], device=DEV),
                batch=batch, stream=torch.cuda.Stream())


def _run_batch(s):
    now = torch.cuda.current_stream()
    s["stream"].wait_stream(now)
    s["batch"].graph_launch(s["H"], s["volumes"], s["stream"])
    now.wait_stream(s["stream"])
    return s["volumes"]


# ---------------------------------------------------------------- training

TRAIN_DIMS = (32, 32, 32)


def _prepare_train(c, seed):
    """Coarse volumes as broad bumps with a brighter shell, the shell's blocks occupied."""
    b = c["batch"]
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    ax = torch.linspace(-1, 1, 32, device=DEV)
    r = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"))
    ctr = torch.rand((b, 3, 1, 1, 1), generator=gen, device=DEV) - 0.5
    rad = 0.2 + 0.2 * torch.rand((b, 1, 1, 1), generator=gen, device=DEV)
    d = (r[None] - ctr).norm(dim=1)
    shell = torch.exp(-((d - rad) / 0.06).square())
    noise = torch.rand(d.shape, generator=gen, device=DEV)
    coarse = (torch.exp(-d.square()) + 0.3 * shell + 0.02 * noise).contiguous()
    model = octree.OccupancyCNN(DEV, seed=seed % 1000)
    X = model.features(coarse, TRAIN_DIMS, b)
    labels = (shell > 0.8).to(torch.uint8).reshape(-1).contiguous()
    return dict(kind="train", model=model, X=X, labels=labels, batch=b)


def _run_train(s):
    m = s["model"]
    loss = m.train_step(s["X"], s["labels"], TRAIN_DIMS, s["batch"], 2e-3, 50.0)
    return {"loss": loss, "gradient": m.flat_G, "weights": m.flat_W}


# ---------------------------------------------------------------- the entry points

def prepare(case, seed):
    return {"dense": _prepare_dense, "host": _prepare_host, "phasor": _prepare_phasor,
            "octree": _prepare_octree, "batch": _prepare_batch,
            "train": _prepare_train}[case["kind"]](case, seed)


def run(state):
    return {"dense": _run_dense, "host": _run_host, "phasor": _run_phasor, "octree": _run_octree,
            "batch": _run_batch, "train": _run_train}[state["kind"]](state)


def work(case):
    k = case["kind"]
    if k == "train":
        v = case["batch"] * 32 ** 3
        acts = (2 + 3 * 16) * 2 + 4  # features, three activations, the logit, kept for backward
        macs = 27 * (2 * 16 + 16 * 16 + 16 * 16 + 16)
        return {"bytes": v * (2 * acts + 1), "flops": 6.0 * v * macs}
    if k == "batch":
        caps = _batch_captures(case)
        rows = sum(_pairs_count(c) * c["T"] for c in caps)
        vox = sum(c["nx"] * c["ny"] * c["nz"] for c in caps)
        return {"bytes": 2 * rows + 4 * vox,
                "flops": UPDATE_FLOPS * sum(_updates(c) for c in caps)}
    if k == "octree":  # the coarse pass and 3% of the fine voxels
        P, v = case["gx"] * case["gy"], case["n"] ** 3
        return {"bytes": 4.0 * (P * case["T"] + v),
                "flops": UPDATE_FLOPS * P * (v / 512 + 0.03 * v)}
    P, v = _pairs_count(case), case["nx"] * case["ny"] * case["nz"]
    if k == "phasor":
        g = _geometry(case)
        taps = int(4 * _wavelength(case) / g["dt"])
        return {"bytes": 4.0 * P * case["T"] + 8.0 * v,
                "flops": (UPDATE_FLOPS + 1) * _updates(case) + 4.0 * P * case["T"] * taps}
    return {"bytes": 4.0 * (P * case["T"] + v), "flops": UPDATE_FLOPS * _updates(case)}


# ---------------------------------------------------------------- the same in 64 bits

def _exact_volume(g, H):
    """Sum over pairs of H[p, bin(v, p)] for every voxel, FP64 geometry and sums."""
    nx, ny, nz = g["n"]
    z = torch.tensor(np.asarray(g["zero"], np.float64), device=DEV)
    inc = torch.tensor(np.asarray(g["inc"], np.float64).reshape(3, 3), device=DEV)
    ax = [torch.arange(k, device=DEV, dtype=torch.float64) for k in (nx, ny, nz)]
    idx = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    v = z + idx @ inc
    cam, las, cw, lw = (f.double() for f in _fields(g["pairs"]))
    P, T = H.shape[0], g["T"]
    t0, dt = float(np.float32(g["t0"])), float(np.float32(g["dt"]))
    out = torch.zeros(v.shape[0], dtype=torch.complex128 if H.is_complex() else torch.float64,
                      device=DEV)
    block = max(1, int(2.5e7) // v.shape[0])
    kept, leg = None, None
    lp = g["pairs"]["laser_point"]
    for p in range(0, P, block):
        q = slice(p, min(P, p + block))
        lq = lp[q]
        if (lq == lq[0]).all():  # one laser point: its leg once
            if kept is None or not (lq[0] == kept).all():
                kept, leg = lq[0], _distance(v, las[p:p + 1])
            d = _distance(v, cam[q]) + leg
        else:
            d = _distance(v, cam[q]) + _distance(v, las[q])
        d += (cw[q] + lw[q] - t0)[:, None]
        b = d.div_(dt).round_().long()
        ok = (b >= 0) & (b < T)
        x = torch.gather(H[q, :T], 1, b.clamp_(0, T - 1))
        out += torch.where(ok, x, torch.zeros((), dtype=x.dtype, device=DEV)).to(out.dtype).sum(0)
    return out.reshape(nx, ny, nz)


def _distance(v, p):
    s = None
    for k in range(3):
        d = (v[None, :, k] - p[:, k, None]).square_()
        s = d if s is None else s.add_(d)
    return s.sqrt_()


def _pulse64(H, c, g):
    """The phasor pulse: K taps of a complex carrier under a Gaussian of sigma 4 wl / 6."""
    wl, dt = np.float32(_wavelength(c)), np.float32(g["dt"])
    K, C = int(np.float32(4) * wl / dt), int(wl / dt)
    sigma = float(np.float32(4) * wl / np.float32(6))
    k = np.arange(1, K + 1, dtype=np.float64)
    tap = np.exp(-(float(dt) * (k - K / 2.0)) ** 2 / (2 * sigma * sigma)) * \
        np.exp(1j * 2 * np.pi * k / C)
    x = H.double().clone()
    x[:, 0] = 0.0  # the convolution leaves out bin 0
    T = H.shape[1]
    n = 1 << (T + K).bit_length()
    spec = torch.fft.fft(torch.from_numpy(tap[::-1].copy()).to(DEV), n)
    out = torch.empty((H.shape[0], T), dtype=torch.complex128, device=DEV)
    for r in range(0, H.shape[0], 1024):
        full = torch.fft.ifft(torch.fft.fft(x[r:r + 1024].to(torch.complex128), n) * spec)
        first = K - 1 - K // 2
        out[r:r + 1024] = full[:, first:first + T]
    return out


def exact(case, seed):
    k = case["kind"]
    if k in ("octree", "train"):
        return None  # a network in 16 bits decides, no value in 64 bits stands for it
    if k == "batch":
        caps, geos = _batch_parts(case)
        if sum(_updates(c) for c in caps) > 8e10:
            return None
        return torch.cat([_exact_volume(g, _transients(g, seed * 1000 + i, points=12).double())
                          .reshape(-1) for i, g in enumerate(geos)])
    if _updates(case) > 8e10:
        return None
    g = _geometry(case)
    if k == "phasor":
        H = _transients(g, seed, peak=None)
        return torch.view_as_real(_exact_volume(g, _pulse64(H, case, g)))
    v = _exact_volume(g, _transients(g, seed).double())
    return v.cpu().numpy() if k == "host" else v
