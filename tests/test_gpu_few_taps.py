"""Phasor pulses of few taps: their own kernel up to 30 taps, and every remainder of the taps by 8
above, bit for bit against the oracle's loop; bound by memory, not by their preparation."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi
from oracle import oracle

pytestmark = pytest.mark.gpu


# T: a CTA of one to four warps with 8 outputs per thread, full and ragged, and two of them
@pytest.mark.parametrize("T,extra", [(5, 0), (256, 1), (257, 0), (511, 2), (700, 0), (1024, 1), (1025, 3)])
def test_few_taps_bit_identical(cuda, T, extra):
    import torch

    dT = 0.001
    H = np.random.default_rng(T).normal(size=(3, T)).astype(np.float32)
    H[1, T // 2] = np.inf
    pitch = T + extra
    dH = torch.zeros((3, pitch), dtype=torch.float32, device=cuda)
    dH[:, :T] = torch.from_numpy(H).to(cuda)
    for K in (4, 5, 7, 8, 17, 29, 30, 31, 32, 33, 34, 35, 36, 37, 38, 39, 40, 515):
        wl = float(np.float32((K + 0.5) * dT / 4))
        assert capi.lib().bpgb_phasor_taps(wl, dT, 4, None, 0) == K
        dO = torch.zeros((3, pitch), dtype=torch.complex64, device=cuda)
        capi.phasor_pulse_device(dH, 3, T, pitch, wl, dT, dO, pitch)
        got = dO.cpu().numpy()
        assert np.array_equal(got[:, :T].view(np.float32), oracle.phasor_pulse(H, wl, dT).view(np.float32),
                              equal_nan=True), K
        assert not got[:, T:].any()


def test_few_taps_cost(cuda):
    """Four taps read each row once and write the field once: 1.5 times a copy of as many bytes
    leaves room (the kernel for many taps took 1.8 times)."""
    import torch

    P, T = 16384, 4096
    H, F = torch.rand((P, T), device=cuda), torch.empty((P, T), dtype=torch.complex64, device=cuda)
    a = torch.empty((3 * P * T // 2,), device=cuda)
    b = torch.empty_like(a)

    def best(f):
        s, e, out = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True), 1e9
        for _ in range(8):
            s.record()
            for _ in range(5):
                f()
            e.record()
            torch.cuda.synchronize()
            out = min(out, s.elapsed_time(e))
        return out

    dT = 0.001
    wl = float(np.float32(4.5 * dT / 4))
    assert best(lambda: capi.phasor_pulse_device(H, P, T, T, wl, dT, F, T)) < 1.5 * best(lambda: b.copy_(a))
