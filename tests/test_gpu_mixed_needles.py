"""Triangle contacts of the mixed form on needles, the short edge at each vertex in turn: every sphere over a needle's face
has the oracle's contact force, by the cooperative pass, the per-particle pass and the pass with tangential history (the
spheres at rest, so that their springs are zero)."""
import numpy as np
import pytest

from metakonga_gb300 import engine, scenes
from metakonga_gb300.layouts import make_params

from .cases import packed_scene
from .test_gpu_mixed import FORCE_TOL, _norm_err
from .test_gpu_mixed_mesh import _oracle_mesh_view

pytestmark = pytest.mark.gpu
R, LENGTH, SIDE, EACH = 0.002, 0.1, 20, 16


def _over_needles(width, seed):
    """400 needles 2 cm apart, each with 16 spheres over its two faces that overlap it by up to 1 % of the radius."""
    rng = np.random.Generator(np.random.MT19937(seed))
    k = SIDE * SIDE
    site = np.stack([np.zeros(k), np.arange(k) % SIDE * 0.02, np.arange(k) // SIDE * 0.02], 1)
    a = rng.uniform(0.0, 2.0 * np.pi, k)
    e = np.tile([1.0, 0.0, 0.0], (k, 1)) + rng.uniform(-0.02, 0.02, (k, 3)) * [0, 1, 1]
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    f = np.stack([np.zeros(k), np.cos(a), np.sin(a)], 1)
    f -= np.sum(f * e, axis=1, keepdims=True) * e
    f /= np.linalg.norm(f, axis=1, keepdims=True)
    skew = rng.uniform(-0.9, 0.9, (k, 1))
    tri = np.stack([site, site + width * (f + skew * e), site + LENGTH * e], axis=1)
    for i in range(k):
        tri[i] = np.roll(tri[i], i % 3, axis=0)
    along = (np.arange(EACH) + 0.5) / EACH * 0.9 + rng.uniform(-0.01, 0.01, (k, EACH))
    across = rng.uniform(0.05, 0.95, (k, EACH)) * (1.0 - along) * width
    side = np.where(np.arange(EACH) % 2 == 0, 1.0, -1.0) * R * (1.0 - 0.01 * rng.uniform(0, 1, (k, EACH)))
    pos = np.empty((k * EACH, 4))
    pos[:, :3] = (site[:, None] + (along * LENGTH)[..., None] * e[:, None] +
                  across[..., None] * (f + skew * e)[:, None] + side[..., None] * np.cross(e, f)[:, None]).reshape(-1, 3)
    pos[:, 3] = R
    sc = packed_scene(n_side=2)
    sc.poly, sc.sphere, sc.vlist = scenes._mesh_arrays(tri)
    sc.poly["id"] = 0
    sc.pmi = np.zeros(1, dtype=scenes.POLYGON_MASS)
    sc.pmi["ep"] = (1.0, 0.0, 0.0, 0.0)
    sc.cp_poly = np.array([sc.cp_pp])
    sc.planes, sc.cp_planes, sc.plane_names = sc.planes[:0], sc.cp_planes[:0], []
    sc.pos = pos
    for key, x in scenes._state(pos).items():
        setattr(sc, key, x)
    sc.params = make_params(np_=pos.shape[0], ncell=16 ** 3, grid=(16,) * 3, dt=1e-6, cell_size=1.5 * LENGTH,
                            world_origin=(-8.0 * LENGTH,) * 3, gravity=(0, 0, 0))
    sc.params["half2dt"] = 0.5e-12
    return sc


@pytest.mark.parametrize("history,mode", [(0, 1), (0, 0), (12, 1)])
@pytest.mark.parametrize("width", [1e-6, 1e-5, 1e-4, 1e-3, 5e-3])
def test_no_needle_contact_is_lost(cuda, oracle, width, mode, history):
    sc = _over_needles(width, seed=int(1e6 * width))
    ds = engine.DeviceScene(sc, mode=engine.MODE_MIXED, tuning={"contact_mode": mode})
    if history:
        ds.set_tangential_history(history)
    f, _ = ds.eval_contacts()
    _, f_ref, _, mag, _ = _oracle_mesh_view(oracle, sc, ds.download())
    assert (np.abs(f_ref).max(axis=1) > 0).mean() > 0.99
    assert _norm_err(f, f_ref, mag, sc.mass, g=0.0) <= FORCE_TOL
    acc = sc.copy()
    ds.step(1, check=True)          # and by the step's own pass, which lists the needles anew
    got = ds.download()
    ds.close()
    oracle.run(acc, 1)
    assert np.array_equal(np.any(got["acc"] != 0.0, axis=1), np.any(acc.acc != 0.0, axis=1))
