"""Stream order of the kernels queued by programmatic dependent launch: passes that follow and
precede other work on the same buffers without a synchronisation, and passes captured behind
copies, memsets and joined streams, give the results of synchronised passes."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi, synthetic

pytestmark = pytest.mark.gpu


def _plan(cuda, kind):
    import torch

    c = synthetic.make_capture("precision_64", seed=3, small=True)
    n = tuple(int(v) for v in c.voxels_per_side)
    pairs = c.pairs.copy()
    opt = {}
    if kind == "exact":
        opt["algo"] = capi.ALGO_EXACT
    elif kind == "split":
        opt["pair_splits"] = 5
    elif kind == "unsplit":
        opt["pair_splits"] = 1
    plan = capi.Plan(pairs, c.T, n, c.zero, c.inc, c.t0, c.deltaT, **opt)
    return c, n, plan, torch.from_numpy(c.H).to(cuda)


@pytest.mark.parametrize("kind", ["split", "unsplit", "exact"])
def test_back_to_back_passes(cuda, kind):
    """Rows rewritten between passes, volumes copied out after each, nothing waits."""
    import torch

    c, n, plan, H = _plan(cuda, kind)
    buf, V = torch.empty_like(H), torch.empty(n, device=cuda)
    scales = [float(k % 7 + 1) for k in range(40)]
    got = []
    for s in scales:
        torch.mul(H, s, out=buf)
        plan.execute(buf, V)
        got.append(V.clone())
        buf.zero_()
    torch.cuda.synchronize()
    ref = {}
    for s in set(scales):
        torch.mul(H, s, out=buf)
        torch.cuda.synchronize()
        plan.execute(buf, V)
        torch.cuda.synchronize()
        ref[s] = V.clone()
    assert all(torch.equal(g, ref[s]) for g, s in zip(got, scales))
    plan.close()


@pytest.mark.parametrize("before", ["nothing", "memset", "copy", "convert", "join"])
def test_captured_passes(cuda, before):
    import torch

    c, n, plan, H = _plan(cuda, "split")
    V, H2, mx = torch.empty(n, device=cuda), torch.zeros_like(H), torch.empty(1, device=cuda)
    plan.execute(H, V)
    torch.cuda.synchronize()
    ref = V.clone()
    V.zero_()
    s, side = torch.cuda.Stream(), torch.cuda.Stream()
    H2.copy_(H)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        rows = H
        if before == "memset":
            V.zero_()
        elif before == "copy":
            H2.copy_(H)
            rows = H2
        elif before == "convert":
            capi.rows_absmax(H, 1, H.numel(), H.numel(), mx, s)
        elif before == "join":
            side.wait_stream(s)
            with torch.cuda.stream(side):
                H2.mul_(1.0)
            V.fill_(1.0)
            s.wait_stream(side)
            rows = H2
        plan.execute(rows, V, s)
        plan.execute(rows, V, s)
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(V, ref)
    plan.close()


def test_conversion_chain(cuda):
    """absmax, conversion, backprojection and rescaling queued in a row, on changing rows."""
    import torch

    c, n, plan, H = _plan(cuda, "split")
    plan.close()
    rows, mx = torch.empty(H.shape, dtype=torch.float16, device=cuda), torch.empty(1, device=cuda)
    V, buf = torch.empty(n, device=cuda), torch.empty_like(H)
    with capi.Plan(c.pairs, c.T, n, c.zero, c.inc, c.t0, c.deltaT, h_dtype=capi.DTYPE_F16,
                   pair_splits=3) as p:
        def one(scale, sync):
            torch.mul(H, scale, out=buf)
            step = torch.cuda.synchronize if sync else (lambda: None)
            step()
            capi.rows_absmax(buf, c.P, c.T, c.T, mx)
            step()
            capi.rows_to_half(buf, c.P, c.T, c.T, capi.DTYPE_F16, rows, c.T, d_absmax=mx, target=16384.0)
            step()
            p.execute(rows, V)
            step()
            capi.volume_scale(V, V.numel(), d_absmax=mx, target=16384.0)
            out = V.clone()
            step()
            return out

        got = [one(1.0 + k, False) for k in range(20)]
        torch.cuda.synchronize()
        assert all(torch.equal(g, one(1.0 + k, True)) for k, g in enumerate(got))


@pytest.mark.parametrize("T,spads,lasers,opt", [
    (1100, (32, 33), None, {}), (1101, (32, 33), None, {"pair_splits": 3}),
    (2051, (29, 18), None, {"pair_splits": 9, "chunk": 7}),
    (1100, (10, 9), (4, 3), {"unfactored": 1, "pair_splits": 5}),
    (1100, (12, 10), (4, 3), {}), (1100, (32, 33), None, {"accum": capi.ACCUM_KAHAN}),
    (1100, (32, 33), None, {"pair_splits": 1}), (1100, (32, 33), None, {"algo": capi.ALGO_EXACT}),
])
def test_host_call_in_parts_equals_a_plan(cuda, T, spads, lasers, opt):
    """Captures large enough to be uploaded in parts: the host call's volume is the plan's, bit
    for bit, on the first call and on repeats with new rows."""
    import torch

    c = synthetic.make_capture("precision_64" if lasers is None else "dense_exhaustive_16", seed=1,
                               render=False, spad_grid=spads, laser_grid=lasers, T=T, deltaT=0.003)
    n, rng = (21, 18, 23), np.random.default_rng(T)
    zero, inc = capi.volume_basis(c.volume_position, c.volume_size, np.uint32(n))
    pitch = (T + 3) // 4 * 4
    assert c.P * T * 4 >= 4 << 20
    rows, V = torch.zeros((c.P, pitch), device=cuda), torch.empty(n, device=cuda)
    with capi.Plan(c.pairs, T, n, zero, inc, c.t0, c.deltaT, h_pitch=pitch, **opt) as plan:
        for _ in range(3):
            H = rng.random((c.P, T), dtype=np.float32)
            rows[:, :T] = torch.from_numpy(H).to(cuda)
            plan.execute(rows, V)
            want = V.cpu().numpy()
            got = capi.backproject_host(H, c.pairs, n, zero, inc, c.t0, c.deltaT, **opt)
            assert np.array_equal(got, want)
