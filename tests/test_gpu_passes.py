"""The elementwise and reduction passes at the edges of their vector paths: rows whose lengths,
pitches and addresses are or are not multiples of 16 bytes, pieces of 16,384 elements, pair
splits around the reductions' segments of 8, volumes with ragged z lines."""
from __future__ import annotations

import numpy as np
import pytest

from backprojector_gb300 import capi, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,T,pitch,out_pitch,shift,special", [
    (1, 1, 1, 1, 0, None), (3, 7, 7, 7, 0, None), (5, 90, 100, 96, 0, "nan"), (4, 64, 64, 64, 1, None),
    (2, 501, 504, 512, 0, "inf"), (3, 8192, 8192, 8192, 0, None), (1, 16385, 16385, 16385, 0, None),
    (2, 40000, 40001, 40008, 0, "-inf"), (7, 33, 36, 33, 0, None),
])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_row_passes(cuda, rows, T, pitch, out_pitch, shift, special, dtype):
    import torch

    rng = np.random.default_rng(rows * T)
    H = np.full((rows, pitch), 1e30, np.float32)  # bins past T must not count
    H[:, :T] = rng.normal(size=(rows, T))
    if special:
        H[rows - 1, T - 1] = float(special)
    flat = torch.zeros(rows * pitch + shift, dtype=torch.float32, device=cuda)
    flat[shift:] = torch.from_numpy(H.reshape(-1)).to(cuda)
    dH = flat[shift:]
    mx = torch.empty(1, dtype=torch.float32, device=cuda)
    capi.rows_absmax(dH, rows, T, pitch, mx)
    want = np.abs(H[:, :T]).max() if special is None else np.float32(np.inf)
    assert mx.item() == want
    tdt, code = ((torch.float16, capi.DTYPE_F16), (torch.bfloat16, capi.DTYPE_BF16))[dtype == "bf16"]
    out = torch.full((rows, out_pitch), 7.0, dtype=tdt, device=cuda)
    capi.rows_to_half(dH, rows, T, pitch, code, out, out_pitch, scale=0.37)
    ref = torch.zeros((rows, out_pitch), dtype=tdt, device=cuda)
    inv = np.float32(1.0) / np.float32(0.37)
    ref[:, :T] = torch.from_numpy(H[:, :T] * inv).to(cuda).to(tdt)
    assert torch.equal(torch.nan_to_num(out.float(), nan=1e9), torch.nan_to_num(ref.float(), nan=1e9))
    n = rows * pitch
    capi.volume_scale(dH, n, scale=0.37)
    np.testing.assert_array_equal(dH.cpu().numpy(), (H.reshape(-1) * np.float32(0.37)))


@pytest.mark.parametrize("splits", [1, 2, 8, 9, 16, 63, 64, 65, 130])
@pytest.mark.parametrize("voxels,cplx,tile", [((21, 20, 23), False, -1), ((17, 9, 18), True, -1),
                                              ((24, 16, 20), False, 13)])
def test_split_sums(cuda, splits, voxels, cplx, tile):
    """Integer rows: sums are exact in any order, so every split count gives one volume, and a
    tile list of every tile gives it too."""
    import torch

    c = synthetic.make_capture("precision_64", seed=4, render=False, spad_grid=(20, 21), T=600,
                               deltaT=0.006)
    rng = np.random.default_rng(1)
    H = rng.integers(0, 1000, (c.P, c.T)).astype(np.float32)
    if cplx:
        H = (H + 1j * rng.integers(0, 1000, (c.P, c.T))).astype(np.complex64)
    zero, inc = capi.volume_basis(c.volume_position, c.volume_size, np.uint32(voxels))
    dH = torch.from_numpy(H).to(cuda)
    opt = dict(h_dtype=capi.DTYPE_C64 if cplx else capi.DTYPE_F32, algo=capi.ALGO_FAST, chunk=3,
               tile=tile)

    def run(s, tiles):
        dV = torch.full(voxels, float("nan"), dtype=dH.dtype, device=cuda)
        with capi.Plan(c.pairs, c.T, voxels, zero, inc, c.t0, c.deltaT, pair_splits=s, **opt) as p:
            info = p.info()
            assert info["pair_splits"] == s
            if tiles:
                n = int(np.prod([-(-v // t) for v, t in zip(voxels, info["tile"])]))
                lst = torch.arange(n, dtype=torch.int32, device=cuda)
                p.execute_tiles(dH, dV, lst, torch.tensor([n], dtype=torch.int32, device=cuda), n)
            else:
                p.execute(dH, dV)
            p.check()
            return dV.cpu().numpy()

    want = run(1, False)
    assert np.array_equal(run(splits, False), want)
    assert np.array_equal(run(splits, True), want)


@pytest.mark.parametrize("coarse,fine", [((1, 1, 1), (3, 1, 5)), ((4, 5, 6), (9, 17, 13)),
                                         ((4, 3, 8), (5, 8, 64)), ((2, 9, 3), (7, 7, 4))])
def test_upsample_edges(cuda, coarse, fine):
    import torch

    rng = np.random.default_rng(2)
    c = rng.normal(size=coarse).astype(np.float32)
    out = torch.full(fine, float("nan"), device=cuda)
    capi.upsample_trilinear(torch.from_numpy(c).to(cuda), coarse, out, fine)
    ref = c.astype(np.float64)
    for a in range(3):
        u = np.arange(fine[a]) * ((coarse[a] - 1) / max(1, fine[a] - 1))
        lo = np.minimum(np.floor(u + 1e-9).astype(int), coarse[a] - 1)
        hi = np.minimum(lo + 1, coarse[a] - 1)
        w = (u - lo).reshape([-1 if k == a else 1 for k in range(3)])
        ref = np.take(ref, lo, a) * (1 - w) + np.take(ref, hi, a) * w
    # FP32 weights are within a few 1e-6 (grid coordinates up to 9), values of order 1
    np.testing.assert_allclose(out.cpu().numpy(), ref, atol=2e-5)


@pytest.mark.parametrize("dtype", ["f32", "bf16", "c64", "c32"])
@pytest.mark.parametrize("tile", [-1, 13])
def test_rows_per_stage(cuda, dtype, tile):
    """Stages of every remainder of the unrolled rows (16, 8, 4, 1) give one volume: integer
    rows, small enough to be exact in 16 bits."""
    import torch

    if tile == 13 and dtype[0] == "c":
        pytest.skip("several tiles per CTA: real rows")
    c = synthetic.make_capture("precision_64", seed=5, render=False, spad_grid=(11, 9), T=512,
                               deltaT=0.007)
    rng = np.random.default_rng(3)
    H = torch.from_numpy(rng.integers(0, 100, (c.P, c.T)).astype(np.float32)).to(cuda)
    if dtype == "c64":
        rows = torch.complex(H, H.flip(1))
    elif dtype == "c32":
        rows = torch.stack([H, H.flip(1)], -1).half().contiguous()
    else:
        rows = H.bfloat16() if dtype == "bf16" else H
    n = (18, 11, 19)
    zero, inc = capi.volume_basis(c.volume_position, c.volume_size, np.uint32(n))
    code = {"f32": capi.DTYPE_F32, "bf16": capi.DTYPE_BF16, "c64": capi.DTYPE_C64,
            "c32": capi.DTYPE_C32}[dtype]
    want = None
    for chunk in (1, 2, 3, 4, 5, 7, 8, 11, 12, 15, 16, 17, 20, 24, 29, 31, 32, 47, 64):
        V = torch.full(n, float("nan"), dtype=torch.complex64 if dtype[0] == "c" else torch.float32,
                       device=cuda)
        with capi.Plan(c.pairs, c.T, n, zero, inc, c.t0, c.deltaT, algo=capi.ALGO_FAST, h_dtype=code,
                       chunk=chunk, tile=tile) as p:
            p.execute(rows, V)
            p.check()
        got = V.cpu().numpy()
        want = got if want is None else want
        assert np.array_equal(got, want), chunk
