"""Calls of one step of a mixed scene: one graph launch that holds the whole call, with the bits of the same steps launched
directly, between longer calls, on moving meshes and scenes that re-bin, and with an emitter."""
import numpy as np
import pytest

from metakonga_gb300 import engine

from .cases import packed_scene, small_hopper
from .cuda_calls import runtime_calls
from .test_gpu_emitter import _stacked
from .test_gpu_gaps import _closing
from .test_gpu_kinematic import _spinning_drum
from .test_gpu_step_graphs import _both

pytestmark = pytest.mark.gpu
CALLS = [(1, 1, 1), (1, 5, 1, 1, 20, 1), (20, 1, 2, 1)]


@pytest.mark.parametrize("make", [packed_scene, small_hopper])
def test_one_launch_a_call(cuda, make):
    d = engine.DeviceScene(make(), mode=engine.MODE_MIXED)
    d.step(1, check=True)
    names = runtime_calls(lambda: [d.step(1) for _ in range(3)])
    d.close()
    names = [x for x in names if "Launch" in x]
    assert names == ["cudaGraphLaunch"] * 3, names


@pytest.mark.parametrize("calls", CALLS)
@pytest.mark.parametrize("speed", [1e-3, 150.0])
def test_spheres(cuda, calls, speed):
    _both(_closing(300, speed, 9), calls)


@pytest.mark.parametrize("calls", CALLS)
def test_walls_history_and_moving_mesh(cuda, calls):
    _both(packed_scene(n_side=6), calls)
    _both(packed_scene(n_side=6), calls, history=True)
    sc = _spinning_drum()
    sc.pmi["omega"] = (0.0, 400.0, 0.0)
    _both(sc, calls, kinematic=True)


def test_emitter(cuda):
    """Steps one at a time across emissions, before and after the graphs of a longer call."""
    got = []
    for calls in ((60,), (1,) * 60, (20,) + (1,) * 20 + (20,)):
        sc, em = _stacked()
        d = engine.DeviceScene(sc, mode=engine.MODE_MIXED)
        d.set_emitter(em["period"], em["groups"], em["active"])
        for n in calls:
            d.step(n, check=True)
        got.append(d.download())
        d.close()
    for k in ("pos", "vel", "omega"):
        assert np.array_equal(got[0][k], got[1][k]) and np.array_equal(got[0][k], got[2][k]), k
