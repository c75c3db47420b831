"""Batches whose lasers x SPADs captures would take different factored forms as plans: half tiles, full
ones where few rows of a window fit a stage (with much or little of the work), and per-pair
captures beside them.

Rows are integers, so sums are exact in any order: a capture's volume must equal its plan's."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi, synthetic

pytestmark = pytest.mark.gpu

# lasers, SPADs, T, voxels, deltaT: windows from one TMA box to several
HALF = [((3, 4), (4, 3), 512, (9, 9, 9), 0.003), ((4, 2), (4, 4), 512, (33, 8, 12), 0.003)]
FULL = [((2, 3), (2, 2), 2048, (17, 10, 18), 0.0007), ((5, 3), (4, 5), 2048, (20, 17, 16), 0.0008)]
WIDE = [((1, 2), (2, 2), 4096, (12, 10, 9), 0.0004), ((4, 5), (5, 4), 512, (33, 17, 20), 0.003)]
PAIRS = [((1, 1), (9, 7), 256, (20, 9, 17), 0.006), ((1, 1), (8, 8), 2048, (10, 12, 7), 0.0008)]


def _capture(lasers, spads, T, voxels, dT):
    c = synthetic.make_capture("dense_exhaustive_16", seed=2, render=False, laser_grid=lasers,
                               spad_grid=spads, T=T, deltaT=dT)
    zero, inc = capi.volume_basis(c.volume_position, c.volume_size, np.uint32(voxels))
    H = np.random.default_rng(T).integers(0, 256, (c.P, T)).astype(np.float32)
    return c, zero, inc, H


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("shapes,opt", [
    (HALF, {}), (FULL, {}), (HALF + FULL, {}), (WIDE + HALF[:1], {}), (FULL + PAIRS, {}),
    (HALF + FULL + PAIRS, {}), (HALF + FULL + PAIRS, {"pair_splits": 3}),
    (HALF + FULL + PAIRS, {"chunk": 5}), (FULL + HALF, {"chunk": 32, "stages": 3}),
    (HALF + FULL + PAIRS, {"unfactored": 1}),
])
def test_batch_equals_plans(cuda, shapes, opt, dtype):
    import torch

    code, tdt = {"f32": (capi.DTYPE_F32, torch.float32), "f16": (capi.DTYPE_F16, torch.float16)}[dtype]
    caps = [(_capture(*s), s[3]) for s in shapes]
    want = []
    for (c, z, i, h), n in caps:
        pitch = (c.T + 7) // 8 * 8
        rows = torch.zeros((c.P, pitch), dtype=tdt, device=cuda)
        rows[:, :c.T] = torch.from_numpy(h).to(cuda).to(tdt)
        dV = torch.empty(n, device=cuda)
        with capi.Plan(c.pairs, c.T, n, z, i, c.t0, c.deltaT, algo=capi.ALGO_FAST, h_dtype=code,
                       h_pitch=pitch, unfactored=opt.get("unfactored", 0)) as p:
            p.execute(rows, dV)
            p.check()
        want.append(dV.cpu().numpy().reshape(-1))
    geo = [dict(pairs=c.pairs, T=c.T, voxels_per_side=n, zero=z, inc=i, t0=c.t0, deltaT=c.deltaT)
           for (c, z, i, _), n in caps]
    for checked in (0, 1):
        with capi.Batch(geo, h_dtype=code, checked=checked, **opt) as b:
            info = b.info()
            H = torch.zeros((info["total_rows"], info["pitch"]), dtype=tdt, device=cuda)
            for ((c, _, _, h), _), r in zip(caps, b.row_offsets):
                H[r:r + c.P, :c.T] = torch.from_numpy(h).to(cuda).to(tdt)
            V = torch.full((info["total_voxels"],), float("nan"), device=cuda)
            b.execute(H, V)
            assert b.check() == 0
            stream = torch.cuda.Stream()
            for _ in range(2):  # the counters start over
                V.fill_(float("nan"))
                torch.cuda.synchronize()
                b.graph_launch(H, V, stream)
                torch.cuda.synchronize()
            got = V.cpu().numpy()
        for k, (w, o) in enumerate(zip(want, b.voxel_offsets)):
            assert np.array_equal(got[o:o + len(w)], w), k


def test_wide_windows_cost_what_their_plans_cost(cuda):
    """Four captures whose 4,096-bin windows leave few rows per stage: the batch takes the plans' form,
    and so about four times a plan (half tiles took twice that)."""
    import torch

    c, z, i, _ = _capture((12, 12), (12, 12), 4096, (48, 48, 48), 0.0004)
    n = (48, 48, 48)

    def best(f):
        s, e, out = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True), 1e9
        for _ in range(6):
            s.record()
            f()
            e.record()
            torch.cuda.synchronize()
            out = min(out, s.elapsed_time(e))
        return out

    rows, V = torch.rand((c.P, c.T), device=cuda), torch.empty(n, device=cuda)
    with capi.Plan(c.pairs, c.T, n, z, i, c.t0, c.deltaT, algo=capi.ALGO_FAST) as p:
        assert p.info()["factored"] == 1 and p.info()["chunk"] < 32
        plan = best(lambda: p.execute(rows, V))
    geo = dict(pairs=c.pairs, T=c.T, voxels_per_side=n, zero=z, inc=i, t0=c.t0, deltaT=c.deltaT)
    with capi.Batch([geo] * 4, h_dtype=capi.DTYPE_F32) as b:
        info = b.info()
        H = torch.rand((info["total_rows"], info["pitch"]), device=cuda)
        V4 = torch.empty(info["total_voxels"], device=cuda)
        assert best(lambda: b.execute(H, V4)) < 1.3 * 4 * plan
