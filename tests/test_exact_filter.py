"""EXACT's choice to drop the range check of its gathers (host code, no GPU): a plan may only do
so when every bin of the reference's expression lies in [0, T), also for volumes far from the
origin, whose FP32 voxel positions lie outside the box of the exact corners."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

from backprojector_gb300 import build, capi, synthetic
from oracle import oracle

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def exact_filter(tmp_path_factory):
    build.build_library()
    d = tmp_path_factory.mktemp("exact_filter")
    exe, lib = d / "exact_filter", build.LIB_PATH.parent
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{build.INCLUDE}", f"-I{build.CSRC}",
                    f"-I{build.CUDA_HOME / 'include'}", str(ROOT / "tests/cpp/exact_filter.cpp"),
                    "-o", str(exe), f"-L{lib}", "-lbpgb300", f"-Wl,-rpath,{lib}"], check=True,
                   capture_output=True, text=True)

    def run(pairs, T, n, zero, inc, t0, dT):
        with open(d / "in.bin", "wb") as f:
            f.write(np.uint32([T, len(pairs), *n]).tobytes())
            f.write(np.float32([*zero, *np.asarray(inc).reshape(-1), t0, dT]).tobytes())
            f.write(pairs.tobytes())
        r = subprocess.run([str(exe), str(d / "in.bin")], check=True, capture_output=True, text=True)
        e, inside = r.stdout.split()
        return float(e), inside == "1"

    return run


def _paths(pairs, lo, hi, farthest):
    out = pairs["laser_wall"].astype(np.float64) + pairs["camera_wall"]
    for k in ("laser_point", "camera_point"):
        p = pairs[k].astype(np.float64)
        q = np.where(np.abs(p - lo) > np.abs(p - hi), lo, hi) if farthest else np.clip(p, lo, hi)
        out = out + np.sqrt(((p - q) ** 2).sum(1))
    return out


@pytest.mark.parametrize("offset", [0.0, 100.0, 1000.0, 5000.0])
@pytest.mark.parametrize("end", ["first", "last"])
def test_inside_means_every_bin_is_in_range(exact_filter, offset, end):
    n, dT = (16, 16, 16), np.float32(0.001)
    inc = np.diag(np.full(3, 0.0317)).astype(np.float32)
    ids = np.arange(int(np.prod(n)))
    claimed = 0
    for seed in range(12):
        rng = np.random.default_rng(seed)
        zero = (offset + rng.uniform(0, 0.1, 3)).astype(np.float32)
        lo = zero.astype(np.float64)
        hi = lo + inc.astype(np.float64).diagonal() * 15
        pairs = np.zeros(12, capi.PAIR_DTYPE)
        for k in ("laser_point", "camera_point"):
            pairs[k] = rng.uniform(lo, hi, (12, 3))
            pairs[k][:, 1] = hi[1] + 1.5
        # the nearest path half a bin and a little inside the window's first bin, or the
        # farthest one as close to the end of its last
        for slack in (0.47, 0.48):
            near, far = _paths(pairs, lo, hi, False).min(), _paths(pairs, lo, hi, True).max()
            if end == "first":
                t0 = np.float32(near + slack * float(dT))
                T = int(np.ceil((far - float(t0)) / float(dT))) + 8
            else:
                T = int(np.ceil((far - near) / float(dT))) + 8
                t0 = np.float32(far - (T - 1 + slack) * float(dT))
            _, inside = exact_filter(pairs, T, n, zero, inc, t0, dT)
            claimed += inside
            if inside:
                b = oracle.bins(pairs, T, n, zero, inc.reshape(-1), float(t0), float(dT), ids, 1)
                assert (b >= 0).all(), (seed, slack)
    if offset == 0.0:
        assert claimed  # the test's own scenes are not all refused


def test_ordinary_capture_needs_no_range_check(exact_filter):
    c = synthetic.make_capture("precision_64", seed=3, small=True)
    far = float(_paths(c.pairs, c.zero, np.float64(c.zero) + np.float64(c.inc).reshape(3, 3).diagonal() *
                       (np.float64(c.voxels_per_side) - 1), True).max())
    T = int((far - c.t0) / c.deltaT) + 3
    t0 = c.t0 if c.t0 < _paths(c.pairs, c.zero, c.zero, False).min() else 0.0
    e, inside = exact_filter(c.pairs, T, tuple(int(v) for v in c.voxels_per_side), c.zero, c.inc,
                             t0, c.deltaT)
    assert e < 0.01 and inside
