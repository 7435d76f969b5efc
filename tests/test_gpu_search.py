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


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 257, 15_999, 16_000, 16_007, 47_999, 48_000, 48_031])
def test_sizes(cuda, oracle, n):
    sc = _bed(n, seed=n)
    f = _both(sc, oracle)
    assert np.abs(f - sc.force).max() > 1e-3


@pytest.mark.parametrize("n,radius", [(900, 0.012), (900, 0.020), (16_100, 0.012), (48_100, 0.012)])
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
