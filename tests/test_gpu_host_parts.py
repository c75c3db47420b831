"""The host call in parts: captures large enough for it give the plan's volume, bit for bit, from
pageable and pinned rows, on the first call and on repeats; small ones are copied at once."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi, synthetic

pytestmark = pytest.mark.gpu


def _scene(spads, lasers, T, n):
    c = synthetic.make_capture("precision_64" if lasers is None else "dense_exhaustive_16", seed=1,
                               render=False, spad_grid=spads, laser_grid=lasers, T=T, deltaT=0.003)
    zero, inc = capi.volume_basis(c.volume_position, c.volume_size, np.uint32(n))
    return c, zero, inc


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("T,spads,lasers,opt,launches", [
    (1101, (64, 64), None, {}, 5), (1100, (64, 64), None, {"pair_splits": 3}, 4),
    (1099, (61, 67), None, {"pair_splits": 9, "chunk": 7}, 5),
    (1100, (64, 64), None, {"pair_splits": 2, "accum": capi.ACCUM_KAHAN}, 3),
    (1101, (16, 16), (4, 4), {"unfactored": 1, "pair_splits": 5}, 5),
    (1100, (64, 64), None, {"pair_splits": 1}, 1), (1100, (16, 16), (4, 4), {"pair_splits": 4}, 2),
])
def test_parts_equal_a_plan(cuda, T, spads, lasers, opt, launches, pinned):
    import torch

    n, rng = (45, 44, 41), np.random.default_rng(T)
    c, zero, inc = _scene(spads, lasers, T, n)
    assert c.P * T * 4 >= 11e6 and c.P * np.prod(n) >= 3e8
    pitch = (T + 3) // 4 * 4
    rows, V = torch.zeros((c.P, pitch), device=cuda), torch.empty(n, device=cuda)
    H = torch.empty((c.P, T), pin_memory=pinned).numpy()
    with capi.Plan(c.pairs, T, n, zero, inc, c.t0, c.deltaT, h_pitch=pitch, **opt) as plan:
        for k in range(3):
            H[:] = rng.random((c.P, T), dtype=np.float32)
            rows[:, :T] = torch.from_numpy(H).to(cuda)
            plan.execute(rows, V)
            want = V.cpu().numpy()
            before = capi.launch_count()
            got = capi.backproject_host(H, c.pairs, n, zero, inc, c.t0, c.deltaT, **opt)
            if k:  # the first call also builds its plan's tables
                assert capi.launch_count() - before == launches
            assert np.array_equal(got, want)


@pytest.mark.parametrize("pinned", [False, True])
def test_small_volumes_are_copied_at_once(cuda, pinned):
    import torch

    n = (16, 16, 16)
    c, zero, inc = _scene((64, 64), None, 1024, n)
    H = torch.rand((c.P, 1024), pin_memory=pinned).numpy()
    first = capi.backproject_host(H, c.pairs, n, zero, inc, c.t0, c.deltaT)
    before = capi.launch_count()
    again = capi.backproject_host(H, c.pairs, n, zero, inc, c.t0, c.deltaT)
    assert capi.launch_count() - before == 2  # the pass and its reduction
    assert np.array_equal(first, again)
