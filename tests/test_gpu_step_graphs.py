"""Steps in graphs (1 to 8 a graph, what follows a due re-binning skipped and made up in the loop) against the same
steps launched one by one (phase timing): the same bits, bodies and re-binnings, at the edges of the graphs' lengths, for
scenes that re-bin never, sometimes and every step."""
import numpy as np
import pytest

from metakonga_gb300 import engine

from .cases import packed_scene
from .test_gpu_gaps import _closing
from .test_gpu_kinematic import _spinning_drum

pytestmark = pytest.mark.gpu
STEPS = [(1,), (2, 1), (3, 5), (8, 1, 7), (9,), (17, 2), (45,)]


def _both(sc, steps, kinematic=False, history=False):
    out = []
    for direct in (False, True):
        d = engine.DeviceScene(sc, mode=engine.MODE_MIXED)
        if history:
            d.set_tangential_history(12)
        if kinematic:
            d.set_kinematic_bodies(True)
        d.set_timing(direct)
        for n in steps:
            d.step(n, check=True)
        st = d.download()
        got = [st[k] for k in ("pos", "vel", "acc", "omega", "alpha")] + [d.rebuilds()[0]]
        if kinematic:
            pmi = d.get_bodies()
            got += [pmi[k] for k in ("origin", "ep", "force", "moment")]
        out.append(got)
        d.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    return out[0][5]


@pytest.mark.parametrize("steps", STEPS)
@pytest.mark.parametrize("speed", [1e-3, 10.0, 150.0])
def test_spheres(cuda, steps, speed):
    n = sum(steps)
    rebuilds = _both(_closing(300, speed, 9), steps)
    if speed == 1e-3:
        assert rebuilds == 1
    elif speed == 150.0 and n > 2:
        assert rebuilds >= n // 2


@pytest.mark.parametrize("steps", STEPS)
def test_history(cuda, steps):
    _both(packed_scene(n_side=6), steps, history=True)


@pytest.mark.parametrize("steps", STEPS)
@pytest.mark.parametrize("spin", [20.0, 400.0, 2_000.0])
def test_moving_mesh(cuda, steps, spin):
    sc = _spinning_drum()
    sc.pmi["omega"] = (0.0, spin, 0.0)
    rebuilds = _both(sc, steps, kinematic=True)
    if spin == 2_000.0 and sum(steps) > 3:
        assert rebuilds > 2
