"""Row passes over many short padded rows: correct at the edges of the rows that share a CTA, and
not far slower than the same elements in one long row."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi

pytestmark = pytest.mark.gpu


# rows that share a CTA (units of 512 to 4,096 elements, whole and cut), a CTA per row, and few long
# rows in pieces of 1,024 to 16,384
@pytest.mark.parametrize("rows,T,pitch,out_pitch", [
    (1000, 1, 2, 8), (777, 2, 3, 2), (1025, 3, 4, 4), (513, 8, 9, 9), (300, 31, 32, 32), (129, 33, 36, 40),
    (70, 127, 128, 128), (65, 129, 132, 136), (40, 512, 516, 512), (33, 1023, 1024, 1025),
    (5, 1025, 1028, 1032), (3, 60001, 60003, 60001), (150, 16385, 16388, 16392),
])
def test_rows_that_share_a_block(cuda, rows, T, pitch, out_pitch):
    import torch

    rng = np.random.default_rng(rows * T)
    H = np.full((rows, pitch), 1e30, np.float32)  # bins past T must not count
    H[:, :T] = rng.normal(size=(rows, T))
    mx = torch.empty(1, device=cuda)
    for r, t in ((0, 0), (rows - 1, T - 1), (rows // 2, T // 2)):
        G = H.copy()
        G[r, t] = -50.0
        dG = torch.from_numpy(G).to(cuda)
        capi.rows_absmax(dG, rows, T, pitch, mx)
        assert mx.item() == 50.0
        out = torch.full((rows, out_pitch), 7.0, dtype=torch.float16, device=cuda)
        capi.rows_to_half(dG, rows, T, pitch, capi.DTYPE_F16, out, out_pitch, scale=0.5)
        want = np.zeros((rows, out_pitch), np.float16)
        want[:, :T] = (G[:, :T] * np.float32(2.0)).astype(np.float16)
        assert np.array_equal(out.cpu().numpy(), want)


def _time(torch, f):
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    f(), f(), f()
    best = float("inf")
    for _ in range(5):
        a.record()
        for _ in range(10):
            f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) / 10)
    return best


@pytest.mark.parametrize("T", [3, 8, 40])
def test_short_rows_cost(cuda, T):
    """Both passes are bound by memory; short rows with a padding element read at most twice the
    sectors, so five times the long row's time leaves room (a CTA per row took 30 to 100 times)."""
    import torch

    rows, pitch = 12_000_000 // T, T + 1
    H, mx = torch.rand((rows, pitch), device=cuda), torch.empty(1, device=cuda)
    out = torch.empty((rows, pitch), dtype=torch.float16, device=cuda)
    n = rows * pitch
    for short, long in (
            (lambda: capi.rows_absmax(H, rows, T, pitch, mx), lambda: capi.rows_absmax(H, 1, n, n, mx)),
            (lambda: capi.rows_to_half(H, rows, T, pitch, capi.DTYPE_F16, out, pitch),
             lambda: capi.rows_to_half(H, 1, n, n, capi.DTYPE_F16, out, n))):
        assert _time(torch, short) < 5.0 * _time(torch, long)
