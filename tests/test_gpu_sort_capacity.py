"""Scenes that sort fewer keys than their scratch was made for, where fewer keys make more tiles (131,072 keys make 128,
131,073 make 65): some of the particles active, and the particles alone on a grid of their own beside a mesh."""
import numpy as np
import pytest

from metakonga_gb300 import engine, scenes

from .cases import packed_scene, small_hopper
from .conftest import force_error

pytestmark = pytest.mark.gpu
STATE = ("pos", "vel", "acc", "omega", "alpha")


def _first(sc, m):
    """The scene of sc's first m particles."""
    part = sc.copy()
    for k in STATE + ("force", "moment", "mass", "inertia"):
        setattr(part, k, np.ascontiguousarray(getattr(sc, k)[:m]))
    part.params["np"] = m
    return part


@pytest.mark.parametrize("mode", [engine.MODE_FP64, engine.MODE_MIXED])
@pytest.mark.parametrize("active", [131_072, 112_700])
def test_active_particles_of_a_larger_scene(cuda, mode, active):
    """132,651 particles, the first of them active, against a scene of those alone: the same bits in the FP64 form, the
    mixed form (whose grid origin comes from all the particles) within its trajectory bands."""
    sc = packed_scene(n_side=51)
    got = []
    for part in (False, True):
        ds = engine.DeviceScene(_first(sc, active) if part else sc, mode=mode)
        if not part:
            ds.set_emitter(0, None, active=active)
        ds.step(3, check=True)
        d = ds.download()
        got.append([d[k] for k in STATE])
        ds.close()
    for a, b, k in zip(*got, STATE):
        if mode == engine.MODE_FP64:
            assert np.array_equal(a[:active], b), k
        elif k in ("pos", "vel"):
            band = 1e-9 if k == "pos" else 1e-4 * np.abs(b).max()
            assert np.abs(a[:active] - b).max() <= band, k
        if k == "pos" or (mode == engine.MODE_FP64 and k in ("vel", "omega")):   # (pairs of floats in the mixed form)
            assert np.array_equal(a[active:], getattr(sc, k)[active:]), k


def test_own_particle_grid_of_a_hopper(cuda, oracle):
    """130,000 particles sorted alone in the scratch of 134,096 entries: positions as the oracle's, forces within the
    FP64 form's 1e-12 of max(|F|, m g) (the pair sums run in another order)."""
    sc = small_hopper(n=130_000)
    assert sc.ntri == 4_096
    ref = sc.copy()
    ds = engine.DeviceScene(sc, mode=engine.MODE_FP64)
    ds.set_particle_grid()
    ds.step(1, check=True)
    got = ds.download()
    ds.close()
    oracle.run(ref, 1)
    assert np.array_equal(got["pos"], ref.pos)
    f, f_ref = got["acc"] * sc.mass[:, None], ref.acc * sc.mass[:, None]
    assert (np.abs(ref.acc - np.array(scenes.GRAVITY)) > 1e-3).any(axis=1).sum() > 1_000
    assert force_error(f, f_ref, sc.mass) <= 1e-12
