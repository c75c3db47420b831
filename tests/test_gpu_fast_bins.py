"""Per-pair plans of every element size read the bins they dump: rows are integers, so sums are exact
in any order and a volume must equal the sum of H at its plan's bins, bit for bit, with and without
the window checks (which test the addresses that the unchecked kernel forms)."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi, synthetic

pytestmark = pytest.mark.gpu

ROWS = {"f32": capi.DTYPE_F32, "f16": capi.DTYPE_F16, "bf16": capi.DTYPE_BF16, "c64": capi.DTYPE_C64,
        "c32": capi.DTYPE_C32}


@pytest.mark.parametrize("rows", list(ROWS))
@pytest.mark.parametrize("spads,T,voxels,dT,opt", [
    ((9, 7), 600, (17, 9, 18), 0.006, {}), ((20, 21), 2048, (21, 20, 23), 0.0008, {"pair_splits": 3}),
    ((12, 11), 600, (9, 16, 33), 0.006, {"accum": capi.ACCUM_KAHAN}), ((8, 9), 90, (12, 10, 14), 0.006, {}),
    ((12, 11), 600, (20, 9, 17), 0.006, {"tile": 10}), ((12, 11), 600, (20, 9, 17), 0.006, {"tile": 13}),
    ((12, 11), 600, (20, 17, 17), 0.006, {"tile": 7}),
])
def test_volume_equals_its_bins(cuda, rows, spads, T, voxels, dT, opt):
    import torch

    cplx = rows in ("c64", "c32")
    c = synthetic.make_capture("precision_64", seed=2, render=False, spad_grid=spads, T=T, deltaT=dT)
    zero, inc = capi.volume_basis(c.volume_position, c.volume_size, np.uint32(voxels))
    rng = np.random.default_rng(T)
    H = rng.integers(0, 256, (c.P, T)).astype(np.float32)
    if cplx:
        H = H + 1j * rng.integers(0, 256, (c.P, T)).astype(np.float32)
    pitch, nvox = (T + 7) // 8 * 8, int(np.prod(voxels))
    dH = torch.zeros((c.P, pitch), dtype=torch.complex64 if cplx else torch.float32, device=cuda)
    dH[:, :T] = torch.from_numpy(H).to(cuda)
    if rows == "c32":
        dH = torch.view_as_real(dH).half().contiguous()
    elif not cplx:
        dH = dH.to({"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}[rows])
    dV = torch.full(voxels, float("nan"), dtype=torch.complex64 if cplx else torch.float32, device=cuda)
    bins = torch.empty((nvox, c.P), dtype=torch.int32, device=cuda)
    for checked in (0, 1):
        try:
            plan = capi.Plan(c.pairs, T, voxels, zero, inc, c.t0, c.deltaT, algo=capi.ALGO_FAST,
                             h_dtype=ROWS[rows], h_pitch=pitch, checked=checked, **opt)
        except capi.BackprojectorError:
            assert "tile" in opt  # presets of four tiles or 16 voxels per thread: not for every row type
            return
        with plan:
            plan.execute(dH, dV)
            assert plan.check() == 0
            plan.dump_bins(np.arange(nvox), bins)
            got = dV.cpu().numpy().reshape(-1)
        b = bins.cpu().numpy()
        want = np.where(b >= 0, H[np.arange(c.P)[None, :], np.maximum(b, 0)], 0).sum(1)
        assert np.array_equal(got, want.astype(got.dtype))
