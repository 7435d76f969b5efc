"""Contact search, pooled groups: the sizes at which a block's warps change (tolerances and cases as in
test_gpu_search.py), and pools that one warp of the block fills alone, over several rounds and chunks."""
import numpy as np
import pytest

from .test_gpu_search import _bed, _both, test_float_lane_counts_agree as float_lanes_agree
from .test_gpu_search import test_triangles as triangles_match

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [15, 16, 17, 32, 33, 4_863, 4_864, 4_865, 4_895, 4_897, 9_728, 9_729])
def test_pool_edges(cuda, oracle, n):
    _both(_bed(n, seed=n), oracle)


@pytest.mark.parametrize("n,first,count", [(64, 28, 12), (4_900, 4_864, 36), (10_100, 8, 24), (48_100, 48_000, 70)])
def test_one_warp_fills_the_pool(cuda, oracle, n, first, count):
    sc = _bed(n, seed=11, pitch=0.02)   # nothing touches but the clump
    rng = np.random.Generator(np.random.MT19937(4))
    sc.pos[first:first + count, :3] = sc.pos[first, :3] + rng.uniform(-0.004, 0.004, (count, 3))
    f = _both(sc, oracle)
    assert (np.abs(f[first:first + count]).max(1) > 1e-3).all()


@pytest.mark.parametrize("n,ntri,nbodies", [(4_863, 1_000, 1), (4_864, 1_000, 2)])
def test_pooltriangles_match(cuda, oracle, n, ntri, nbodies):
    triangles_match(cuda, oracle, n, ntri, nbodies)


@pytest.mark.parametrize("filler", [27_450, 27_520])
def test_float_pool_lines(cuda, filler):
    float_lanes_agree(cuda, filler)
