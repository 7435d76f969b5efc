"""Mixed contact passes visit only the gap classes that the largest displacement since the list build can close, and
the contact view quantises positions with integer instructions.  Pairs at every gap up to the skin, closing within the
run, give the bits of the per-particle pass (which visits every particle), alone and batched; forces of slight
overlaps at coordinates of every magnitude follow the oracle."""
import numpy as np
import pytest

from metakonga_gb300 import engine, scenes
from metakonga_gb300.layouts import make_params

from .test_gpu_mixed import FORCE_TOL, _norm_err, _oracle_view

pytestmark = pytest.mark.gpu


def _pairs(pos, vel, dt, cell, side):
    sc = scenes.settle_box(n_side=2)
    sc.pos = pos
    for key, val in scenes._state(pos).items():
        setattr(sc, key, val)
    sc.vel[:] = vel
    o = pos[:, :3].min(0) - 2 * cell
    sc.params = make_params(np_=pos.shape[0], ncell=side ** 3, grid=(side,) * 3, dt=dt, cell_size=cell,
                            world_origin=tuple(o), gravity=(0, 0, 0))
    sc.params["half2dt"] = 0.5 * dt * dt
    sc.planes = sc.planes[:0]
    sc.cp_planes = sc.cp_planes[:0]
    sc.plane_names = []
    return sc


def _closing(n, speed, seed):
    """n pairs of 5 mm spheres at gaps from a slight overlap to just over the skin (0.1 r), closing at up to `speed`."""
    rng = np.random.Generator(np.random.MT19937(seed))
    r = 0.005
    site = np.stack(np.unravel_index(np.arange(n), (20, 20, 20)), -1) * 0.03
    gap = np.linspace(-1e-5, 0.11 * r, n)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    v = d * (rng.uniform(0.2, 0.5, (n, 1)) * speed)
    pos = np.empty((2 * n, 4))
    pos[0::2, :3], pos[1::2, :3] = site, site + d * (2 * r + gap)[:, None]
    pos[:, 3] = r
    vel = np.empty((2 * n, 3))
    vel[0::2], vel[1::2] = v, -v
    return _pairs(pos, vel, 1e-5, 2 * r, 128)


def _state(d):
    out = d.download()
    return [out[k] for k in ("pos", "vel", "acc", "omega", "alpha")]


# the speed covers no class, a few classes, and several re-binnings in the run
@pytest.mark.parametrize("n,speed", [(1, 1.0), (700, 1e-3), (700, 0.4), (3_000, 1.5), (3_000, 20.0)])
def test_closing_gaps_same_bits(cuda, n, speed):
    sc, other = _closing(n, speed, n), _closing(211, 0.6, 5)
    got = []
    for mode in (0, 1):
        d = engine.DeviceScene(sc, mode=engine.MODE_MIXED, tuning={"contact_mode": mode})
        d.step(45, check=True)
        got.append(_state(d))
        d.close()
    ds = [engine.DeviceScene(s, mode=engine.MODE_MIXED) for s in (other, sc)]
    b = engine.Batch(ds)
    b.step(45, check=True)
    got.append(_state(ds[1]))
    b.close()
    for d in ds:
        d.close()
    if speed >= 0.4 and n > 1:
        assert (np.abs(got[0][2]) > 0).any() and not np.array_equal(got[0][1], sc.vel)
    for x, y, z in zip(*got):
        assert np.array_equal(x, y) and np.array_equal(x, z)


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_slight_overlaps_at_every_magnitude(cuda, oracle, sign):
    # x of the first sphere: zero, subnormal, and 2^-40 .. 2^1 m, dense in mantissa bits and with trailing zeros
    rng = np.random.Generator(np.random.MT19937(3))
    x0 = np.concatenate([[0.0, 5e-324], 2.0 ** np.arange(-40, 2), 2.0 ** np.arange(-40, 2) * rng.uniform(1, 2, 42),
                         (rng.integers(1, 1 << 20, 40) + 0.5) * 2.0 ** -36])
    n = x0.size
    ri, rj = rng.uniform(0.005, 0.0075, (2, n))   # (separations in 31 bits of the fixed point: the force's range)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    depth = 10.0 ** rng.uniform(-8, -6, n)
    pos = np.empty((2 * n, 4))
    pos[0::2, 0] = sign * x0
    pos[0::2, 1:3] = np.stack([np.arange(n) % 12, np.arange(n) // 12], -1) * 0.3
    pos[1::2, :3] = pos[0::2, :3] + d * (ri + rj - depth)[:, None]
    pos[0::2, 3], pos[1::2, 3] = ri, rj
    sc = _pairs(pos, np.zeros((2 * n, 3)), 1e-9, 0.081, 128)
    ds = engine.DeviceScene(sc, mode=engine.MODE_MIXED)
    for steps in (0, 2):   # the view that the upload writes, and the advance's
        if steps:
            ds.step(steps, check=True)
        f, _ = ds.eval_contacts()
        pairs, f_ref, _, mag = _oracle_view(oracle, sc, ds.download())
        assert len(pairs) >= 2 * n * 0.99
        assert _norm_err(f, f_ref, mag, sc.mass, g=0.0) <= FORCE_TOL
    ds.close()
