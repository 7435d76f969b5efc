"""The cooperative contact passes take 4 to 32 listed particles a warp by the list's length.  At the edges (one run a
warp, 32 particles a run, the next round of runs) they give the same bits as the per-particle pass (which the oracle tests pin), alone and batched."""
import numpy as np
import pytest

from metakonga_gb300 import engine

from .test_gpu_search import _bed

pytestmark = pytest.mark.gpu


def _scene(n, seed):
    sc = _bed(n, radius=0.0056, seed=seed)
    sc.params["dt"] = 1e-5
    sc.params["half2dt"] = 0.5e-10
    return sc


def _run(sc, mode, steps=4, evaluate=True):
    # (an evaluation builds the lists where the particles are; without one the first step does, after its drift)
    d = engine.DeviceScene(sc, mode=engine.MODE_MIXED, tuning={"contact_mode": mode})
    out = list(d.eval_contacts()) if evaluate else []
    d.step(steps, check=True)
    out += [d.download()[k] for k in ("pos", "vel", "acc", "omega", "alpha")]
    d.close()
    return out


@pytest.mark.parametrize("n", [1, 3, 4, 5, 257, 9_728, 9_729, 38_912, 38_913, 77_825, 90_001])
def test_run_sizes_same_bits(cuda, n):
    sc = _scene(n, n)
    a, b = _run(sc, 0), _run(sc, 1)
    assert np.abs(a[0]).max() > 0
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("sizes", [(5, 3_000), (9_000, 10_457, 300), (19_000, 19_913), (30_000, 40_000, 1)])
def test_batch_run_sizes_same_bits(cuda, sizes):
    scs = [_scene(n, 100 + k) for k, n in enumerate(sizes)]
    alone = [_run(sc, 1, evaluate=False) for sc in scs]
    ds = [engine.DeviceScene(sc, mode=engine.MODE_MIXED) for sc in scs]
    b = engine.Batch(ds)
    b.step(4, check=True)
    for d, want in zip(ds, alone):
        got = d.download()
        for k, w in zip(("pos", "vel", "acc", "omega", "alpha"), want):
            assert np.array_equal(got[k], w)
    b.close()
    for d in ds:
        d.close()
