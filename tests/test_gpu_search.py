"""The FP64 contact search (FP32 near tests, contacts collected per warp)
against the oracle where it can go wrong: the lane counts it chooses by size
and their remainders, more contacts than a particle's slots, a slip of exactly
zero, coordinates far from the origin, and a grid so small that the 27 cells
repeat.  Tolerance as in test_gpu_contact.py: 1e-12 of max(|F_ref|, m g), the
last-place differences of x sqrt(x) and the device log."""
import numpy as np
import pytest
import torch

from metakonga_gb300 import dem, scenes
from metakonga_gb300.layouts import make_params

from .cases import packed_scene
from .conftest import force_error

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _bed(n, radius=0.0056, pitch=0.011, seed=0, shift=0.0, slip=True, grid=128, slab=0):
    """n spheres on a jittered lattice of `pitch`, `slab` sites thick (0: a cube)."""
    rng = np.random.Generator(np.random.MT19937(seed))
    side = int(np.ceil((n / slab) ** 0.5)) if slab else int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(np.arange(side), np.arange(side), np.arange(slab or side), indexing="ij"), -1)
    pos = np.empty((n, 4))
    pos[:, :3] = g.reshape(-1, 3)[:n] * pitch + rng.uniform(-0.0004, 0.0004, (n, 3)) + shift
    pos[:, 3] = radius
    sc = packed_scene(n_side=2)
    sc.pos = pos
    for k, v in scenes._state(pos).items():
        setattr(sc, k, v)
    if slip:
        sc.vel[:] = rng.normal(0.0, 0.05, (n, 3))
        sc.omega[:] = rng.normal(0.0, 5.0, (n, 3))
    sc.params = make_params(np_=n, ncell=grid ** 3, grid=(grid,) * 3, dt=1e-5, cell_size=2 * radius,
                            world_origin=(-0.1 + shift,) * 3, gravity=(0, 0, -9.81))
    sc.planes, names = scenes.box_walls(pos[:, :3].min(0) - 0.0054, pos[:, :3].max(0) + 0.0054, lid=True)
    sc.cp_planes = np.array([sc.cp_pp] * len(names))
    return sc


def _both(sc, oracle):
    h, ix, cs, ce, so = oracle.detection(sc.params, sc.pos)
    f, m = sc.force.copy(), sc.moment.copy()
    oracle.p2p(sc.params, sc.pos, sc.vel, sc.omega, f, m, sc.mass, so, cs, ce, sc.cp_pp)
    for w in range(sc.planes.shape[0]):
        oracle.plane(sc.params, sc.planes[w:w + 1], sc.pos, sc.vel, sc.omega, f, m, sc.mass, sc.cp_planes[w:w + 1])
    sim = dem.DemSimulation()
    sim.initialize(sc)
    sim.dtor.detection(sim.dpos, None, sim.np, 0)
    assert np.array_equal(sim.dtor.sortedID().cpu().numpy().view(np.uint32), so)
    sim.cm.runCollision(sim.dpos, sim.dvel, sim.davel, sim.dmass, sim.dforce, sim.dmoment, sim.dtor.sortedID(),
                        sim.dtor.cellStart(), sim.dtor.cellEnd(), sim.np)
    torch.cuda.synchronize()
    r = sc.pos[:, 3:4]
    assert force_error(sim.dforce.cpu().numpy(), f, sc.mass) <= TOL
    assert force_error(sim.dmoment.cpu().numpy() / r, m / r, sc.mass) <= TOL
    return f


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 257, 9_999, 10_000, 10_007, 47_999, 48_000, 48_031])
def test_sizes(cuda, oracle, n):
    sc = _bed(n, seed=n)
    f = _both(sc, oracle)
    assert np.abs(f - sc.force).max() > 1e-3


@pytest.mark.parametrize("n,radius", [(900, 0.012), (900, 0.020), (10_100, 0.012), (48_100, 0.012)])
def test_more_contacts_than_slots(cuda, oracle, n, radius):
    """Deep overlaps: some 30 to 120 contacts a sphere, so a round ends several times."""
    _both(_bed(n, radius=radius, seed=7, slab=12), oracle)


@pytest.mark.parametrize("shift", [3.0, -700.0, 1.0e5])
def test_far_from_the_origin(cuda, oracle, shift):
    _both(_bed(2_000, seed=3, shift=shift), oracle)


def test_zero_slip(cuda, oracle):
    """Spheres at rest: the contact before's tangential force (zero) is carried."""
    _both(_bed(1_500, seed=4, slip=False), oracle)


def test_repeated_cells(cuda, oracle):
    """Two cells an axis: the 27 cells of a particle are the same eight, each visited several times."""
    _both(_bed(300, seed=5, grid=2), oracle)


def test_radii_zero_and_not_finite(cuda, oracle):
    """A point, and a sphere whose velocity is not a number, leave the others' forces as the oracle's."""
    sc = _bed(700, seed=6)
    sc.pos[3, 3] = 0.0
    sc.vel[11] = np.nan
    h, ix, cs, ce, so = oracle.detection(sc.params, sc.pos)
    f, m = sc.force.copy(), sc.moment.copy()
    oracle.p2p(sc.params, sc.pos, sc.vel, sc.omega, f, m, sc.mass, so, cs, ce, sc.cp_pp)
    sim = dem.DemSimulation()
    sim.initialize(sc)
    sim.dtor.detection(sim.dpos, None, sim.np, 0)
    sim.cm.cpp.cuda_collision(sim.dpos, sim.dvel, sim.davel, sim.dmass, sim.dforce, sim.dmoment, sim.dtor.sortedID(),
                              sim.dtor.cellStart(), sim.dtor.cellEnd(), sim.np)
    g = sim.dforce.cpu().numpy()
    assert np.array_equal(np.isnan(g), np.isnan(f)) and np.isnan(f).any()
    ok = ~np.isnan(f).any(axis=1)
    assert force_error(g[ok], f[ok], sc.mass[ok]) <= TOL


def _soup(n, ntri, nbodies, seed, big=0.08):
    """n spheres among random triangles of nbodies bodies: ordinary ones, large ones, and slivers down to
    1e-9 of their length wide; most spheres are put on a triangle's face, edge or vertex."""
    rng = np.random.Generator(np.random.MT19937(seed))
    a = rng.uniform(-0.3, 0.3, (ntri, 3))
    size = np.where(np.arange(ntri) % 5 == 0, big, 0.015)[:, None]
    u, v = rng.normal(size=(2, ntri, 3))
    u *= size / np.linalg.norm(u, axis=1, keepdims=True)
    v *= size / np.linalg.norm(v, axis=1, keepdims=True)
    thin = np.arange(ntri) % 7 == 3
    v[thin] = u[thin] * 0.6 + v[thin] * 10.0 ** rng.uniform(-9, -2, (thin.sum(), 1))
    tri = np.stack([a, a + u, a + v], axis=1)
    sc = packed_scene(n_side=2)
    sc.poly, sc.sphere, sc.vlist = scenes._mesh_arrays(tri)
    sc.sphere = np.nan_to_num(sc.sphere)
    sc.poly["id"] = np.arange(ntri) % nbodies
    sc.pmi = np.zeros(nbodies, dtype=scenes.POLYGON_MASS)
    sc.pmi["ep"] = (1.0, 0.0, 0.0, 0.0)
    sc.pmi["vel"] = rng.normal(0.0, 0.05, (nbodies, 3))
    sc.pmi["omega"] = rng.normal(0.0, 1.0, (nbodies, 3))
    sc.cp_poly = np.array([sc.cp_pp] * nbodies)
    w = rng.dirichlet((0.5, 0.5, 0.5), n)
    t = rng.integers(0, ntri, n)
    pos = np.empty((n, 4))
    pos[:, 3] = rng.uniform(0.002, 0.004, n)
    pos[:, :3] = np.einsum("ij,ijk->ik", w, tri[t]) + rng.normal(0.0, 0.0025, (n, 3))
    sc.pos = pos
    for k, x in scenes._state(pos).items():
        setattr(sc, k, x)
    sc.vel[:] = rng.normal(0.0, 0.05, (n, 3))
    sc.omega[:] = rng.normal(0.0, 5.0, (n, 3))
    sc.params = make_params(np_=n, ncell=64 ** 3, grid=(64,) * 3, dt=1e-5, cell_size=0.03, world_origin=(-1.0,) * 3,
                            gravity=(0, 0, -9.81))
    return sc


@pytest.mark.parametrize("n,ntri,nbodies", [(1, 40, 1), (5, 60, 2), (3_001, 2_000, 1), (2_000, 2_000, 3),
                                            (2_000, 1_000, 7), (10_003, 1_500, 1), (48_003, 1_500, 1)])
def test_triangles(cuda, oracle, n, ntri, nbodies):
    sc = _soup(n, ntri, nbodies, seed=n + ntri)
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
    assert force_error(got, f, sc.mass) <= TOL
    assert np.array_equal(np.abs(got - sc.force).max(axis=1) > 0, np.abs(f - sc.force).max(axis=1) > 0)
    assert n < 100 or (np.abs(f - sc.force).max(axis=1) > 0).mean() > 0.3
    scale = np.abs(f - sc.force).sum() + 1e-300
    b = mesh.bodies()
    assert np.abs(b["force"] - pmi["force"]).max() <= TOL * scale
    assert np.abs(b["moment"] - pmi["moment"]).max() <= TOL * scale


@pytest.mark.parametrize("filler", [9_700, 47_700])
def test_float_lane_counts_agree(cuda, filler):
    """The single precision pair and wall contacts of the reference-pinned fixture (test_gpu_fp32.py) are the
    same bits when spheres far away, which touch nothing, make the search use fewer lanes a particle."""
    import os

    from metakonga_gb300._lib import call
    from .test_gpu_fp32 import GOLDEN, _dev, _raw_dev, _rec, _set_params
    from metakonga_gb300.layouts import CONTACT_PROPERTY_F, PARAMS_F, PLANE_F

    d = np.load(os.path.join(GOLDEN, "f32_packed_512_walls.npz"))
    _set_params(d)
    nc, n0 = int(_rec(d["params_f"], PARAMS_F)["ncell"][0]), d["in_pos"].shape[0]
    planes, cps = _raw_dev(d["planes"]).view(-1, PLANE_F.itemsize), _raw_dev(d["cp_planes"]).view(-1, CONTACT_PROPERTY_F.itemsize)
    cp = _raw_dev(d["cp_pp"])
    got = []
    for extra in (0, filler):
        side = int(np.ceil(max(extra, 1) ** (1 / 3)))
        far = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:extra] * 0.013 + 5.0
        S = {k: np.asarray(d["in_" + k]) for k in ("pos", "vel", "omega", "force", "moment", "mass")}
        add = {"pos": np.concatenate([far, np.full((extra, 1), 0.005)], 1), "mass": np.ones(extra)}
        S = {k: _dev(np.concatenate([v, add.get(k, np.zeros((extra, 3)))]).astype(np.float32)) for k, v in S.items()}
        n = n0 + extra
        h, ix, so = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3))
        cs, ce = (torch.zeros(nc, dtype=torch.int32, device="cuda") for _ in range(2))
        call("xd_calculate_hash_and_index_f", h.data_ptr(), ix.data_ptr(), S["pos"].data_ptr(), n, 0)
        call("xd_reorder_and_find_cell_start_f", h.data_ptr(), ix.data_ptr(), cs.data_ptr(), ce.data_ptr(), so.data_ptr(), n, nc, 0)
        args = [S[k].data_ptr() for k in ("pos", "vel", "omega", "force", "moment", "mass")]
        call("xd_calculate_p2p_f", 1, *args, so.data_ptr(), cs.data_ptr(), ce.data_ptr(), cp.data_ptr(), n, 0)
        for w in range(planes.shape[0]):
            call("xd_plane_contact_force_f", 1, planes[w].data_ptr(), *args, n, cps[w].data_ptr(), 0)
        torch.cuda.synchronize()
        got.append([S[k].cpu().numpy()[:n0] for k in ("force", "moment")])
    assert np.abs(got[0][0] - d["in_force"]).max() > 0
    for a, b in zip(*got):
        assert np.array_equal(a, b)
