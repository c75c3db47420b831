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


def _scan(P, seed=3):
    """Pairs that do not factor: laser and SPAD scanned together at a fixed distance."""
    rng = np.random.default_rng(seed)
    p = np.zeros(P, capi.PAIR_DTYPE)
    p["camera_point"][:, 0] = rng.uniform(-0.5, 0.5, P)
    p["camera_point"][:, 2] = rng.uniform(-0.5, 0.5, P)
    p["laser_point"] = p["camera_point"] + np.float32([0.05, 0.0, 0.01])
    p["camera_wall"] = rng.uniform(0.5, 0.9, P)
    p["laser_wall"] = rng.uniform(0.5, 0.9, P)
    return p


def _check(cuda, n, P, T, t0, dT, cplx):
    zero = np.float32([-0.25, 0.35, -0.25])
    inc = np.diag(0.5 / np.maximum(1, np.array(n) - 1)).astype(np.float32).reshape(-1)
    got, want, info, _ = _volume_and_bins(cuda, _scan(P), T, n, zero, inc, t0, dT, cplx)
    assert np.array_equal(got, want)
    return info


# the edges of the filtered kernel's 4 x 4 x 16 tiles; pairs up to sixteen splits
@pytest.mark.parametrize("n,P,splits", [
    ((3, 3, 15), 40, 1), ((4, 4, 16), 64, 1), ((5, 5, 17), 65, 1), ((4, 3, 32), 128, 1),
    ((3, 5, 33), 257, 2), ((5, 4, 31), 2048, 16), ((2, 3, 17), 2300, 16),
])
@pytest.mark.parametrize("cplx", [False, True])
def test_filtered_tiles(cuda, n, P, splits, cplx):
    info = _check(cuda, n, P, 600, 1.5, 0.005, cplx)
    assert tuple(info["tile"]) == (4, 4, 16) and info["threads"] == 64
    assert info["pair_splits"] == splits


# bins so fine that no quotient is trusted, and bins where a small launch would wait for its
# marks: the edges of the direct kernel's 4 x 8 x 8 tiles and of its 256 staged pairs
@pytest.mark.parametrize("T,t0,dT", [(4096, 1.9, 1e-6), (6000, 1.5, 3e-4)])
@pytest.mark.parametrize("n,P,splits", [
    ((1, 1, 1), 1, 1), ((3, 7, 9), 63, 1), ((4, 8, 8), 128, 2), ((5, 9, 7), 255, 3),
    ((4, 7, 17), 257, 4), ((5, 8, 8), 1025, 16), ((3, 9, 16), 4200, 16),
])
@pytest.mark.parametrize("cplx", [False, True])
def test_direct_tiles(cuda, n, P, splits, T, t0, dT, cplx):
    info = _check(cuda, n, P, T, t0, dT, cplx)
    # the legs of the one voxel in the volume's corner are short: a bound of 0.0036 bins at 0.3 mm
    filtered = n == (1, 1, 1) and dT == 3e-4
    assert tuple(info["tile"]) == ((4, 4, 16) if filtered else (4, 8, 8))
    assert info["threads"] == (64 if filtered else 256) and info["pair_splits"] == splits
