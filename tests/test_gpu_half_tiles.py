"""Half tiles past the volume's edge: extents of 1 to 4 voxels beyond whole tiles along the voxel lines
leave the second half of the last tiles without work, in plans, tile lists and batches.

Rows are integers, so sums are exact in any order: volumes must equal the sum of H at the plan's
dumped bins."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi, synthetic

pytestmark = pytest.mark.gpu


def _capture(voxels):
    c = synthetic.make_capture("dense_exhaustive_16", seed=2, render=False, laser_grid=(3, 4),
                               spad_grid=(4, 5), T=512, deltaT=0.012)  # narrow windows: half tiles
    zero, _ = capi.volume_basis(c.volume_position, c.volume_size, np.uint32([8, 8, 8]))
    inc = np.diag(np.full(3, 0.02)).astype(np.float32).reshape(-1)
    return c, zero, inc, np.random.default_rng(5).integers(0, 256, (c.P, c.T)).astype(np.float32)


@pytest.mark.parametrize("depth", [2, 3, 4, 5, 8, 9, 12, 13, 20])
@pytest.mark.parametrize("tile", [-1, 0, 1])
def test_depths(cuda, depth, tile):
    import torch

    voxels = (17, depth, 21) if tile != 1 else (17, 9, depth)
    c, zero, inc, H = _capture(voxels)
    dH, nvox = torch.from_numpy(H).to(cuda), int(np.prod(voxels))
    bins = torch.empty((nvox, c.P), dtype=torch.int32, device=cuda)
    for splits in (0, 1, 3):
        dV = torch.full(voxels, float("nan"), device=cuda)
        with capi.Plan(c.pairs, c.T, voxels, zero, inc, c.t0, c.deltaT, algo=capi.ALGO_FAST, tile=tile,
                       pair_splits=splits) as p:
            info = p.info()
            n = int(np.prod([-(-v // t) for v, t in zip(voxels, info["tile"])]))
            assert info["factored"] == 1 and info["grid"] == 2 * n * info["pair_splits"]
            p.execute(dH, dV)
            assert p.check() == 0
            p.dump_bins(np.arange(nvox), bins)
            b = bins.cpu().numpy()
            want = np.where(b >= 0, H[np.arange(c.P)[None, :], np.maximum(b, 0)], 0).sum(1)
            assert np.array_equal(dV.cpu().numpy().reshape(-1), want.astype(np.float32))
            dV.fill_(float("nan"))
            p.execute_tiles(dH, dV, torch.arange(n, dtype=torch.int32, device=cuda),
                            torch.tensor([n], dtype=torch.int32, device=cuda), n)
            assert p.check() == 0
            assert np.array_equal(dV.cpu().numpy().reshape(-1), want.astype(np.float32))
    geo = dict(pairs=c.pairs, T=c.T, voxels_per_side=voxels, zero=zero, inc=inc, t0=c.t0, deltaT=c.deltaT)
    with capi.Batch([geo, geo], h_dtype=capi.DTYPE_F32, tile=tile) as bt:
        info = bt.info()
        rows = torch.zeros((info["total_rows"], info["pitch"]), device=cuda)
        for r in bt.row_offsets:
            rows[r:r + c.P, :c.T] = dH
        V = torch.full((info["total_voxels"],), float("nan"), device=cuda)
        bt.execute(rows, V)
        assert bt.check() == 0
        got = V.cpu().numpy()
    for o in bt.voxel_offsets:
        assert np.array_equal(got[o:o + nvox], want.astype(np.float32))


def test_a_batch_makes_no_units_for_them(cuda):
    units = {}
    for depth in (12, 16):
        voxels = (16, depth, 16)
        c, zero, inc, _ = _capture(voxels)
        geo = dict(pairs=c.pairs, T=c.T, voxels_per_side=voxels, zero=zero, inc=inc, t0=c.t0,
                   deltaT=c.deltaT)
        with capi.Batch([geo], h_dtype=capi.DTYPE_F32, pair_splits=2) as b:
            units[depth] = b.info()["work_units"]
    assert units == {12: 6, 16: 8}  # 3 and 4 half tiles x 2 pair ranges
