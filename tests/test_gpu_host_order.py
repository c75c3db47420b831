"""The host call reads its rows after the work queued before it in the legacy default stream, and
in the streams that order themselves with it, as a synchronous copy from them does: a buffer
that such work still fills gives the volume of the filled buffer, whatever the capture's size
and whether the memory is pinned."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from backprojector_gb300 import capi, synthetic

pytestmark = pytest.mark.gpu

LARGE, SMALL = (64, 64), (8, 8)  # 4,096 and 64 rows: in parts, and as one copy


def _scene(spads):
    c = synthetic.make_capture("precision_64", seed=1, render=False, spad_grid=spads, T=2048)
    n = (64, 64, 64)
    zero, inc = capi.volume_basis(c.volume_position, c.volume_size, np.uint32(n))
    H = np.random.default_rng(4).random((c.P, c.T), dtype=np.float32)

    def call(rows):
        return capi.backproject_host(rows, c.pairs, n, zero, inc, c.t0, c.deltaT)

    return call, H


def _queue_long_copies(torch, cuda, stream):
    """About 10 ms of device copies."""
    a = torch.empty(1 << 30, dtype=torch.uint8, device=cuda)
    b = torch.empty_like(a)
    with torch.cuda.stream(stream):
        for _ in range(24):
            b.copy_(a, non_blocking=True)
    return a, b


def _cudart():
    for name in ("libcudart.so.13", "libcudart.so"):
        try:
            return C.CDLL(name)
        except OSError:
            continue
    pytest.skip("no CUDA runtime library to load")


@pytest.mark.parametrize("spads", [LARGE, SMALL])
@pytest.mark.parametrize("where", ["default", "blocking"])
def test_pinned_rows_still_being_copied(cuda, spads, where):
    import torch

    call, H = _scene(spads)
    want = call(H)
    pinned, dH = torch.zeros(H.shape, pin_memory=True), torch.from_numpy(H).to(cuda)
    torch.cuda.synchronize()
    if where == "default":
        stream = torch.cuda.default_stream()
    else:  # a stream of the runtime's default kind, which the default stream waits for
        rt, ptr = _cudart(), C.c_void_p()
        assert rt.cudaStreamCreate(C.byref(ptr)) == 0
        stream = torch.cuda.ExternalStream(ptr.value)
    keep = _queue_long_copies(torch, cuda, stream)
    with torch.cuda.stream(stream):
        pinned.copy_(dH, non_blocking=True)
    got = call(pinned.numpy())
    torch.cuda.synchronize()
    del keep
    assert np.array_equal(got, want)


@pytest.mark.parametrize("spads", [LARGE, SMALL])
def test_pageable_rows_written_by_a_queued_host_function(cuda, spads):
    import torch

    call, H = _scene(spads)
    want = call(H)
    rows, rt = np.zeros_like(H), _cudart()
    torch.cuda.synchronize()
    keep = _queue_long_copies(torch, cuda, torch.cuda.default_stream())
    fill = C.CFUNCTYPE(None, C.c_void_p)(lambda _: C.memmove(rows.ctypes.data, H.ctypes.data, H.nbytes))
    assert rt.cudaLaunchHostFunc(C.c_void_p(1), fill, None) == 0  # 1: the legacy default stream
    got = call(rows)
    torch.cuda.synchronize()
    del keep
    assert np.array_equal(got, want)
