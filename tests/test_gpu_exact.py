"""EXACT against its own bins: the kernel that filters updates by a cheap quotient must read
the bin the reference's expression gives for every update (bpgb_plan_dump_bins evaluates that
expression alone).

Rows are integers small enough that every sum stays below 2^24, so sums are exact in any
order and equal bins mean equal volumes, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi

pytestmark = pytest.mark.gpu


def _pairs(P, seed):
    """Pairs that do not factor: laser and SPAD scanned together at a fixed distance."""
    rng = np.random.default_rng(seed)
    p = np.zeros(P, capi.PAIR_DTYPE)
    p["camera_point"][:, 0] = rng.uniform(-0.5, 0.5, P)
    p["camera_point"][:, 2] = rng.uniform(-0.5, 0.5, P)
    p["laser_point"] = p["camera_point"] + np.float32([0.05, 0.0, 0.01])
    p["camera_wall"] = rng.uniform(0.5, 0.9, P)
    p["laser_wall"] = rng.uniform(0.5, 0.9, P)
    return p


# volumes: one voxel, the edges of the 4 x 8 x 8 tiles; pairs: the edges of the groups of 32
# and 64 and of the pair splits; windows that cover every path and ones that cut it at both
# ends; steps so fine that no cheap quotient is trusted
@pytest.mark.parametrize("n,P,T,t0,dT,cplx", [
    ((1, 1, 1), 1, 600, 1.5, 0.005, False),
    ((4, 8, 8), 31, 600, 1.5, 0.005, False),
    ((5, 9, 17), 32, 600, 1.5, 0.005, False),
    ((3, 7, 15), 33, 600, 1.5, 0.005, True),
    ((8, 16, 8), 64, 600, 1.5, 0.005, False),
    ((9, 8, 9), 65, 100, 2.0, 0.005, False),
    ((9, 8, 9), 127, 1000, 1.5, 0.003, False),
    ((6, 17, 10), 300, 101, 2.1, 0.004, True),
    ((12, 12, 12), 1153, 1000, 1.5, 0.003, False),
    ((6, 5, 9), 70, 4096, 1.9, 1e-6, False),
    ((6, 5, 9), 257, 60000, 1.4, 5e-5, True),
])
def test_exact_volume_equals_its_bins(cuda, n, P, T, t0, dT, cplx):
    import torch

    pairs = _pairs(P, 3)
    rng = np.random.default_rng(P)
    H = rng.integers(0, 1000, (P, T)).astype(np.float32)
    if cplx:
        H = (H + 1j * rng.integers(0, 1000, (P, T))).astype(np.complex64)
    zero = np.float32([-0.25, 0.35, -0.25])
    inc = np.diag(0.5 / np.maximum(1, np.array(n) - 1)).astype(np.float32).reshape(-1)
    dH = torch.from_numpy(H).to(cuda)
    dV = torch.full(n, float("nan"), dtype=dH.dtype, device=cuda)
    nvox = int(np.prod(n))
    bins = torch.empty((nvox, P), dtype=torch.int32, device=cuda)
    with capi.Plan(pairs, T, n, zero, inc, t0, dT,
                   h_dtype=capi.DTYPE_C64 if cplx else capi.DTYPE_F32) as plan:
        assert plan.info()["algo"] == "exact"
        plan.execute(dH, dV)
        plan.dump_bins(np.arange(nvox), bins)
        got = dV.cpu().numpy().reshape(-1)
    b = bins.cpu().numpy()
    want = np.where(b >= 0, H[np.arange(P)[None, :], np.maximum(b, 0)], 0).sum(
        axis=1, dtype=np.complex128 if cplx else np.float64)
    assert np.array_equal(got.astype(want.dtype), want)
