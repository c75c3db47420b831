"""Factored lasers x SPADs plans at the edges of their blocks: SPAD counts that end a block of
8 after 4, few lasers, half tiles past the volume's edge, stages of few rows (both forms), and
batches whose captures stage different window widths.

Rows are integers, so sums are exact in any order: a volume must equal the sum of H at the
plan's own dumped bins, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi, synthetic

pytestmark = pytest.mark.gpu


def _capture(lasers, spads, T, voxels, dT):
    c = synthetic.make_capture("dense_exhaustive_16", seed=2, render=False, laser_grid=lasers,
                               spad_grid=spads, T=T, deltaT=dT)
    zero, inc = capi.volume_basis(c.volume_position, c.volume_size, np.uint32(voxels))
    rng = np.random.default_rng(T)
    H = rng.integers(0, 256, (c.P, T)).astype(np.float32)
    return c, zero, inc, H


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("lasers,spads,T,voxels,dT,opt", [
    ((2, 1), (2, 2), 512, (8, 8, 8), 0.003, {}),          # fewer SPADs than a block
    ((3, 3), (2, 6), 512, (17, 9, 5), 0.003, {}),         # 12 SPADs: the last block holds 4
    ((3, 5), (4, 5), 512, (16, 12, 20), 0.003, {}),       # half tiles past the y edge
    ((5, 3), (4, 4), 2048, (9, 11, 10), 0.0008, {}),      # wide windows: few rows per stage
    ((5, 3), (4, 7), 512, (12, 10, 33), 0.003, {"chunk": 32}),
    ((5, 3), (4, 7), 512, (12, 10, 33), 0.003, {"chunk": 5, "pair_splits": 3}),
    ((3, 3), (4, 3), 100, (12, 10, 14), 0.003, {}),       # bins past the row's end
])
def test_factored_volume_equals_its_bins(cuda, lasers, spads, T, voxels, dT, opt, dtype):
    import torch

    c, zero, inc, H = _capture(lasers, spads, T, voxels, dT)
    nvox = int(np.prod(voxels))
    pitch = (T + 7) // 8 * 8
    rows = torch.zeros((c.P, pitch), device=cuda)
    rows[:, :T] = torch.from_numpy(H).to(cuda)
    if dtype == "f16":
        rows = rows.half()
    dV = torch.full(voxels, float("nan"), device=cuda)
    bins = torch.empty((nvox, c.P), dtype=torch.int32, device=cuda)
    for checked in (0, 1):
        with capi.Plan(c.pairs, T, voxels, zero, inc, c.t0, c.deltaT, algo=capi.ALGO_FAST,
                       h_dtype=capi.DTYPE_F16 if dtype == "f16" else capi.DTYPE_F32,
                       h_pitch=pitch, checked=checked, **opt) as plan:
            assert plan.info()["factored"] == 1
            plan.execute(rows, dV)
            assert plan.check() == 0
            plan.dump_bins(np.arange(nvox), bins)
            got = dV.cpu().numpy().reshape(-1)
        b = bins.cpu().numpy()
        want = np.where(b >= 0, H[np.arange(c.P)[None, :], np.maximum(b, 0)], 0).sum(1)
        assert np.array_equal(got, want.astype(np.float32))


def test_batch_of_uneven_windows_equals_plans(cuda):
    """Per-pair and factored captures whose windows span one to several TMA boxes."""
    import torch

    shapes = [((1, 1), (9, 7), 256, (20, 9, 17), 0.006), ((3, 4), (4, 3), 512, (9, 9, 9), 0.003),
              ((1, 1), (8, 8), 2048, (10, 12, 7), 0.0008), ((4, 2), (4, 4), 1024, (33, 8, 12), 0.0015),
              ((2, 3), (2, 2), 2048, (8, 10, 11), 0.0007)]
    caps = [(_capture(*s), s) for s in shapes]
    for code, tdt in ((capi.DTYPE_F32, torch.float32), (capi.DTYPE_F16, torch.float16)):
        geo = [dict(pairs=c.pairs, T=c.T, voxels_per_side=s[3], zero=z, inc=i, t0=c.t0,
                    deltaT=c.deltaT) for (c, z, i, _), s in caps]
        with capi.Batch(geo, h_dtype=code, checked=1) as b:
            info = b.info()
            H = torch.zeros((info["total_rows"], info["pitch"]), dtype=tdt, device=cuda)
            for (c, _, _, h), r in zip((k[0] for k in caps), b.row_offsets):
                H[r:r + c.P, :c.T] = torch.from_numpy(h).to(cuda).to(tdt)
            V = torch.full((info["total_voxels"],), float("nan"), device=cuda)
            b.execute(H, V)
            assert b.check() == 0
            got = V.cpu().numpy()
        for ((c, z, i, h), s), o in zip(caps, b.voxel_offsets):
            n = int(np.prod(s[3]))
            pitch = (c.T + 7) // 8 * 8
            rows = torch.zeros((c.P, pitch), dtype=tdt, device=cuda)
            rows[:, :c.T] = torch.from_numpy(h).to(cuda).to(tdt)
            dV = torch.empty(s[3], device=cuda)
            with capi.Plan(c.pairs, c.T, s[3], z, i, c.t0, c.deltaT, algo=capi.ALGO_FAST,
                           h_dtype=code, h_pitch=pitch) as p:
                p.execute(rows, dV)
                p.check()
            assert np.array_equal(got[o:o + n], dV.cpu().numpy().reshape(-1))
