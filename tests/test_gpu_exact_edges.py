"""EXACT where its choices change: volumes far from the origin whose paths end within a window's
first and last half bin.  Rows are integers, so sums are exact in any order: a volume must equal
the sum of H at the plan's dumped bins, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi

pytestmark = pytest.mark.gpu


def _volume_and_bins(cuda, pairs, T, n, zero, inc, t0, dT, cplx, spare=0):
    """The plan's volume and the sums of H at its dumped bins; `spare` rows that no update may
    read surround H."""
    import torch

    P, rng = len(pairs), np.random.default_rng(T)
    H = rng.integers(0, 1000, (P, T)).astype(np.float32)
    if cplx:
        H = (H + 1j * rng.integers(0, 1000, (P, T))).astype(np.complex64)
    dH = torch.full((P + 2 * spare, T), 1e6, dtype=torch.complex64 if cplx else torch.float32,
                    device=cuda)
    rows = dH[spare:spare + P]
    rows.copy_(torch.from_numpy(H))
    dV = torch.full(n, float("nan"), dtype=dH.dtype, device=cuda)
    nvox = int(np.prod(n))
    bins = torch.empty((nvox, P), dtype=torch.int32, device=cuda)
    with capi.Plan(pairs, T, n, zero, inc, t0, dT, algo=capi.ALGO_EXACT,
                   h_dtype=capi.DTYPE_C64 if cplx else capi.DTYPE_F32) as plan:
        info = plan.info()
        plan.execute(rows, dV)
        plan.dump_bins(np.arange(nvox), bins)
        got = dV.cpu().numpy().reshape(-1)
    b = bins.cpu().numpy()
    want = np.where(b >= 0, H[np.arange(P)[None, :], np.maximum(b, 0)], 0).sum(
        axis=1, dtype=np.complex128 if cplx else np.float64)
    return got.astype(want.dtype), want, info, b


@pytest.mark.parametrize("end,seed", [("first", 5), ("first", 45), ("last", 7), ("last", 15)])
@pytest.mark.parametrize("cplx", [False, True])
def test_tight_window_far_from_the_origin(cuda, end, seed, cplx):
    n, dT, rng = (16, 16, 16), np.float32(0.001), np.random.default_rng(seed)
    inc = np.diag(np.full(3, 0.0317)).astype(np.float32)
    zero = (5000.0 + rng.uniform(0, 0.1, 3)).astype(np.float32)
    lo = zero.astype(np.float64)
    hi = lo + inc.astype(np.float64).diagonal() * 15
    pairs = np.zeros(12, capi.PAIR_DTYPE)
    for k in ("laser_point", "camera_point"):
        pairs[k] = rng.uniform(lo, hi, (12, 3))
        pairs[k][:, 1] = hi[1] + 1.5

    def paths(farthest):
        out = 0.0
        for k in ("laser_point", "camera_point"):
            p = pairs[k].astype(np.float64)
            q = np.where(np.abs(p - lo) > np.abs(p - hi), lo, hi) if farthest else np.clip(p, lo, hi)
            out = out + np.sqrt(((p - q) ** 2).sum(1))
        return out

    near, far = paths(False).min(), paths(True).max()
    T = int(np.ceil((far - near) / float(dT))) + 8
    t0 = near + 0.47 * float(dT) if end == "first" else far - (T - 1 + 0.47) * float(dT)
    got, want, _, b = _volume_and_bins(cuda, pairs, T, n, zero, inc.reshape(-1), float(np.float32(t0)),
                                       float(dT), cplx, spare=1)
    assert (b < 0).any()  # some updates lie outside the window
    assert np.array_equal(got, want)
