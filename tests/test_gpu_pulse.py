"""The phasor pulse at the edges of its tiling, bit for bit against the oracle's loop: 8
outputs per thread, segments of at most 1,024 outputs, taps staged 512 at a time, 16-byte
stores only where the rows allow them."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,K,extra", [
    (1, 4, 0), (7, 9, 1), (8, 8, 0), (9, 15, 2), (255, 7, 1), (256, 64, 0), (1023, 503, 1),
    (1024, 511, 0), (1025, 512, 1), (2050, 513, 2), (1500, 1030, 0),
])
def test_pulse_edges_bit_identical(cuda, T, K, extra):
    import torch

    dT = 0.001
    wl = float(np.float32((K + 0.5) * dT / 4))
    assert capi.lib().bpgb_phasor_taps(wl, dT, 4, None, 0) == K
    rng = np.random.default_rng(T)
    H = rng.normal(size=(3, T)).astype(np.float32)
    ref = oracle.phasor_pulse(H, wl, dT)
    pitch = T + extra
    dH = torch.zeros((3, pitch), dtype=torch.float32, device=cuda)
    dH[:, :T] = torch.from_numpy(H).to(cuda)
    dO = torch.zeros((3, pitch), dtype=torch.complex64, device=cuda)
    capi.phasor_pulse_device(dH, 3, T, pitch, wl, dT, dO, pitch)
    got = dO.cpu().numpy()
    assert np.array_equal(got[:, :T], ref)
    assert not got[:, T:].any()
