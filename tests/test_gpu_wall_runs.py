"""Wall runs take 8 listed particles, in a batch with a long front 16: at the edges (one run a warp, the line) a layer of spheres between two planes gets the bits of the per-particle pass, alone and batched."""
import numpy as np
import pytest

from metakonga_gb300 import engine

from .test_gpu_runs import _run
from .test_gpu_search import _bed

pytestmark = pytest.mark.gpu


def _layer(n, seed):
    sc = _bed(n, radius=0.0056, seed=seed, slab=1)
    sc.params["dt"] = 1e-5
    sc.params["half2dt"] = 0.5e-10
    return sc


@pytest.mark.parametrize("n", [9, 19_457, 77_824, 77_825, 80_001])
def test_layers_same_bits(cuda, n):
    sc = _layer(n, n)
    a, b = _run(sc, 0), _run(sc, 1)
    assert np.abs(a[0]).max() > 0
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("sizes", [(9_000, 17), (50_000, 17, 27_807), (50_000, 17, 27_808), (60_000, 30_001)])
def test_batched_layers_same_bits(cuda, sizes):
    scs = [_layer(n, 7 + n) for n in sizes]
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
