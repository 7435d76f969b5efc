"""FP64 triangle contacts on needles, the short edge at each vertex in turn (the FP32 test that selects them must not
lose one where its barycentric coordinates cancel): the same spheres touch as the oracle's, and with its forces."""
import numpy as np
import pytest
import torch

from metakonga_gb300 import dem, scenes
from metakonga_gb300.layouts import make_params

from .cases import packed_scene
from .conftest import force_error

pytestmark = pytest.mark.gpu
TOL = 1e-12   # as in test_gpu_search.py


def _needles(n, ntri, length, width, seed):
    """n spheres of 3 mm over the face of needles (30 to 150 degrees at the short edge), overlapping by up to 1 % of the radius."""
    rng = np.random.Generator(np.random.MT19937(seed))
    unit = lambda m: (lambda a: a / np.linalg.norm(a, axis=1, keepdims=True))(rng.normal(size=(m, 3)))
    e, f = unit(ntri), unit(ntri)
    f -= np.sum(f * e, axis=1, keepdims=True) * e
    f /= np.linalg.norm(f, axis=1, keepdims=True)
    o = rng.uniform(-0.2, 0.2, (ntri, 3)) - 0.5 * length * e
    skew = rng.uniform(-0.9, 0.9, (ntri, 1))
    tri = np.stack([o, o + width * (f + skew * e), o + length * e], axis=1)
    for k in range(ntri):
        tri[k] = np.roll(tri[k], k % 3, axis=0)
    sc = packed_scene(n_side=2)
    sc.poly, sc.sphere, sc.vlist = scenes._mesh_arrays(tri)
    sc.poly["id"] = 0
    sc.pmi = np.zeros(1, dtype=scenes.POLYGON_MASS)
    sc.pmi["ep"] = (1.0, 0.0, 0.0, 0.0)
    sc.cp_poly = np.array([sc.cp_pp])
    t = rng.integers(0, ntri, n)
    w = rng.dirichlet((1.0, 1.0, 1.0), n)
    d = np.cross(e, f)[t] * np.where(rng.uniform(size=(n, 1)) < 0.5, 1.0, -1.0)   # over the face, where the barycentrics count
    pos = np.empty((n, 4))
    pos[:, 3] = 0.003
    pos[:, :3] = np.einsum("ij,ijk->ik", w, tri[t]) + d * 0.003 * (1.0 - 0.01 * rng.uniform(0, 1, (n, 1)))
    sc.pos = pos
    for k, x in scenes._state(pos).items():
        setattr(sc, k, x)
    sc.vel[:] = rng.normal(0.0, 0.05, (n, 3))
    sc.params = make_params(np_=n, ncell=16 ** 3, grid=(16,) * 3, dt=1e-5, cell_size=1.5 * length,
                            world_origin=(-8.0 * length,) * 3, gravity=(0, 0, -9.81))
    return sc


@pytest.mark.parametrize("length,width", [(1.0, 1e-5), (1.0, 3e-6), (3.0, 1e-5), (0.3, 3e-6), (0.3, 1e-3), (0.1, 0.02)])
def test_no_needle_contact_is_lost(cuda, oracle, length, width):
    n = 8_000
    sc = _needles(n, 90, length, width, seed=int(1e6 * length) + int(1e7 * width))
    h, ix, cs, ce, so = oracle.detection(sc.params, sc.pos, sc.sphere)
    f, m, pmi = sc.force.copy(), sc.moment.copy(), sc.pmi.copy()
    oracle.polygon(sc.params, sc.poly, sc.sphere, pmi, sc.pos, sc.vel, sc.omega, f, m, sc.mass, so, cs, ce, sc.cp_poly)
    d = {k: dem.to_dev(getattr(sc, k)) for k in ("pos", "vel", "omega", "force", "moment", "mass")}
    grid = [torch.from_numpy(np.ascontiguousarray(x).view(np.int32).copy()).cuda() for x in (so, cs, ce)]
    dem.set_symbolic_parameter(sc.params)
    mesh = dem.ContactParticlesPolygonObjects(sc.poly, sc.sphere, sc.vlist, sc.pmi, sc.cp_poly)
    mesh.cuda_collision(d["pos"], d["vel"], d["omega"], d["mass"], d["force"], d["moment"], *grid, n)
    torch.cuda.synchronize()
    got = d["force"].cpu().numpy()
    touch = np.abs(f - sc.force).max(axis=1) > 0
    assert touch.mean() > 0.9
    assert np.array_equal(np.abs(got - sc.force).max(axis=1) > 0, touch)
    assert force_error(got, f, sc.mass) <= TOL
