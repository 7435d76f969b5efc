"""The gap classes of the mixed list against the oracle, which knows none: pairs that all close as fast as the fastest, so that
the displacement since the build only just allows for them, from gaps on both sides of every class's edge and densely in
between.  After calls of every length the spheres with a force, and the recorded pairs, are those that touch."""
import numpy as np
import pytest

from metakonga_gb300 import engine

from .test_gpu_gaps import _pairs
from .test_gpu_mixed import _oracle_view, _pairset

pytestmark = pytest.mark.gpu
R, SKIN = 0.005, 0.1 * 0.005


def _closing_at_one_speed(speed):
    edges = SKIN * (np.arange(1, 9) / 8.0) ** 2
    gap = np.concatenate([np.linspace(-1e-6, 1.02 * SKIN, 1_500)] +
                         [edges * (1.0 + s * e) for s in (-1.0, 1.0) for e in (1e-6, 1e-4, 1e-3, 1e-2, 3e-2)])
    n = gap.size
    rng = np.random.Generator(np.random.MT19937(2))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    site = np.stack(np.unravel_index(np.arange(n), (20, 20, 20)), -1) * 0.03
    pos = np.empty((2 * n, 4))
    pos[0::2, :3], pos[1::2, :3] = site, site + d * (2 * R + gap)[:, None]
    pos[:, 3] = R
    vel = np.empty((2 * n, 3))
    vel[0::2], vel[1::2] = d * speed, -d * speed
    return _pairs(pos, vel, 1e-5, 2 * R, 128)


def _check(oracle, sc, ds):
    st = ds.download()
    want = _pairset(_oracle_view(oracle, sc, st)[0])
    assert _pairset(np.flatnonzero(np.any(st["acc"] != 0.0, axis=1))[:, None]) == {(i,) for p in want for i in p}
    assert _pairset(ds.pair_list()) == want
    return len(want)


# 0.1, 0.5 and 5 m/s: 1, 5 and 50 um a step towards each other of a skin of 500
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("speed,calls", [(0.1, (1, 2, 1, 5, 8, 9, 17, 24)), (0.5, (1,) * 48),
                                         (5.0, (1, 2, 1, 5, 8, 9, 17, 24))])
def test_every_contact_is_visited(cuda, oracle, mode, speed, calls):
    sc = _closing_at_one_speed(speed)
    ds = engine.DeviceScene(sc, mode=engine.MODE_MIXED, tuning={"contact_mode": mode})
    seen = []
    for k in calls:
        ds.step(k, check=True)
        seen.append(_check(oracle, sc, ds))
    ds.close()
    assert max(seen) > 100 and len(set(seen)) > 3


def test_every_contact_is_visited_in_a_batch(cuda, oracle):
    scs = [_closing_at_one_speed(s) for s in (0.5, 0.2)]
    ds = [engine.DeviceScene(s, mode=engine.MODE_MIXED) for s in scs]
    b = engine.Batch(ds)
    for k in (1, 3, 8, 20, 13):
        b.step(k, check=True)
        for sc, d in zip(scs, ds):
            assert _check(oracle, sc, d) > 0
    b.close()
    for d in ds:
        d.close()
