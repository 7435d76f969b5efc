"""The legacy interface's hash takes the cells by the same FP32 estimate as the current one: the same hashes, coordinates on
cell faces included, in about the same time (the divisions that the estimate saves take eight times as long)."""
import numpy as np
import pytest
import torch

from metakonga_gb300 import dem
from metakonga_gb300._lib import call, ptr
from metakonga_gb300.layouts import LEGACY_PARAMS, make_params

pytestmark = pytest.mark.gpu
SIDE, CELL, ORIGIN = 128, 0.008, -0.5


def _time(f, reps=20):
    for _ in range(3):
        f()
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    best = 1e9
    for _ in range(5):
        a.record()
        for _ in range(reps):
            f()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b) / reps)
    return best


def test_same_hashes_in_the_same_time(cuda):
    n = 2_000_000
    rng = np.random.Generator(np.random.MT19937(1))
    pos = np.zeros((n, 4))
    pos[:, :3] = rng.uniform(ORIGIN - 0.1, ORIGIN + 0.1 + SIDE * CELL, (n, 3))
    pos[: n // 64, :3] = ORIGIN + CELL * rng.integers(0, SIDE, (n // 64, 3))   # on faces
    p = np.zeros(1, LEGACY_PARAMS)
    p["np"], p["ncell"], p["grid"], p["dt"], p["cell_size"] = n, SIDE ** 3, SIDE, 1e-5, CELL
    p["world_origin"] = ORIGIN
    call("xd_legacy_set_symbolic_parameter", p.ctypes.data)
    dem.set_symbolic_parameter(make_params(np_=n, ncell=SIDE ** 3, grid=(SIDE,) * 3, dt=1e-5, cell_size=CELL,
                                           world_origin=(ORIGIN,) * 3, gravity=(0, 0, -9.81)))
    dpos = dem.to_dev(pos)
    out = [[torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2)] for _ in range(2)]
    s = dem.stream_handle()
    # (np = 1: the legacy call hashes the block's particles and sorts none)
    calls = [lambda: call("xd_legacy_calculate_hash_and_index", ptr(out[0][0]), ptr(out[0][1]), ptr(dpos), 1, s),
             lambda: call("xd_calculate_hash_and_index", ptr(out[1][0]), ptr(out[1][1]), ptr(dpos), n, s)]
    t = [_time(f) for f in calls]
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert t[0] < 3.0 * t[1], t
