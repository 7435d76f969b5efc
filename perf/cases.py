"""The calls whose speed this framework is judged by, as a user's program makes them.

Three ways in are measured:

* the calls of the reference's own interface on device arrays (metakonga_gb300.dem and the single
  precision twins of the C ABI): a whole step of a small settle, the cell grid, the contact layers
  with and without a triangle mesh, a whole step in float;
* one scene kept on the device (metakonga_gb300.engine.DeviceScene), as a job: its state is uploaded
  from pinned memory, advanced, and downloaded, in the FP64 and in the mixed form;
* many scenes at once: a batch of hoppers (engine.Batch) and a server's tick over unequal scenes
  (engine.step_many), as jobs too.

Beds are packings of spheres with small overlaps (a periodic cell relaxed from random points, tiled
into the container), because almost all of a run is spent with the particles in contact; boxes that
are still falling together are clouds with few contacts.  Everything is made from the seed.
"""
import functools
import math

import numpy as np
import torch

from metakonga_gb300 import dem, engine, scenes
from metakonga_gb300._lib import call
from metakonga_gb300.layouts import CONTACT_PROPERTY_F, PARAMS_F, PLANE_F, to_single

FIELDS = ("pos", "vel", "acc", "omega", "alpha")
WIDTH = {"pos": 4, "vel": 3, "acc": 3, "omega": 3, "alpha": 3, "force": 3, "moment": 3, "mass": 1, "inertia": 1}


def listed():
    return [
        # the reference's CPU-runnable settle, one step through its class interface: latency and launches
        {"name": "step_settle_8000", "kind": "step", "shape": "settle", "n": 8000},
        # the grid of a full-size box: hash, sort and cell ranges of a million particles
        {"name": "grid_box_1m", "kind": "grid", "shape": "loose", "n": 1_000_000},
        # FP64 particle and wall contacts of a mid-size bed (the drop-in library's main cost)
        {"name": "contacts_box_120k", "kind": "contacts", "shape": "bed", "n": 120_989},
        # FP64 contacts on the coarse grid that a triangle mesh imposes: the median hopper
        {"name": "contacts_hopper_17k", "kind": "contacts", "shape": "hopper", "n": 17_159, "orifice": 8.0, "fric": 0.4},
        # a whole step in single precision (the reference's float build)
        {"name": "step_float_100k", "kind": "float", "shape": "bed", "n": 100_003},
        # the settle as an FP64 job
        {"name": "job_fp64_settle_8000", "kind": "job", "mode": "fp64", "shape": "settle", "n": 8000, "steps": 100},
        # the settle as a mixed-form job: a step costs its launches
        {"name": "job_settle_8000", "kind": "job", "mode": "mixed", "shape": "settle", "n": 8000, "steps": 400},
        # the largest hopper of the discharge batch, a packed bed on triangles
        {"name": "job_hopper_199k", "kind": "job", "mode": "mixed", "shape": "hopper", "n": 199_583, "steps": 100,
         "orifice": 8.0, "fric": 0.4},
        # a million spheres still falling: the state's traffic
        {"name": "job_box_1m", "kind": "job", "mode": "mixed", "shape": "loose", "n": 1_000_000, "steps": 200},
        # the drum turning on the device, its mesh of 20,480 triangles moved every step
        {"name": "job_drum_500k", "kind": "job", "mode": "mixed", "shape": "drum", "n": 500_000, "steps": 100},
        # independent hoppers discharging as one batch
        {"name": "batch_hoppers_12", "kind": "batch", "count": 12, "steps": 50},
        # a server's tick: unequal boxes and hoppers side by side
        {"name": "served_8", "kind": "served", "count": 8, "steps": 50},
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    kind = rng.choice(["step", "grid", "contacts", "float", "job64", "job", "job", "batch", "served"])
    hopper = {"orifice": round(rng.uniform(6.0, 12.0), 3), "fric": round(rng.uniform(0.2, 0.6), 3)}
    if kind == "step":
        return {"kind": "step", "shape": "settle", "n": size(1_000, 60_000)}
    if kind == "grid":
        return {"kind": "grid", "shape": "loose", "n": size(4_000, 1_000_000)}
    if kind == "contacts":
        if rng.random() < 0.5:
            return {"kind": "contacts", "shape": "bed", "n": size(2_000, 200_000)}
        return dict(hopper, kind="contacts", shape="hopper", n=size(2_000, 20_000))
    if kind == "float":
        return {"kind": "float", "shape": "bed", "n": size(2_000, 200_000)}
    if kind == "job64":
        return {"kind": "job", "mode": "fp64", "shape": rng.choice(["settle", "bed", "loose"]), "n": size(1_000, 60_000),
                "steps": rng.choice([20, 50, 100])}
    if kind == "job":
        shape = rng.choice(["settle", "bed", "loose", "hopper", "hopper", "drum"])
        lo, hi = {"settle": (1_000, 60_000), "bed": (2_000, 200_000), "loose": (1_000, 1_000_000),
                  "hopper": (2_000, 200_000), "drum": (60_000, 500_000)}[shape]
        case = {"kind": "job", "mode": "mixed", "shape": shape, "n": size(lo, hi), "steps": rng.choice([50, 100])}
        return dict(hopper, **case) if shape == "hopper" else case
    return {"kind": kind, "count": rng.randint(3, 12 if kind == "batch" else 8), "steps": rng.choice([20, 50])}


# ------------------------------------------------------------------ inputs

def _rng(seed, *more):
    return np.random.Generator(np.random.MT19937([int(seed) & 0x7FFFFFFF, *more]))


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


@functools.lru_cache(maxsize=4)
def _cell(seed, rmin, rmax, loose=False):
    """A periodic cell of spheres (centres, radii, side): 1,500 random points relaxed until about 4.5
    neighbours of each overlap it by some 0.05 % of the radius, as in a settled bed; or, loose, a falling
    cloud in which a third have a neighbour within half a millimetre and few touch one."""
    n, rng = 1500, _rng(seed, 1)
    r = rng.uniform(rmin, rmax, n)
    side = ((4.0 / 3.0) * math.pi * (r ** 3).sum() / (0.16 if loose else 0.58)) ** (1.0 / 3.0)
    x = torch.tensor(rng.uniform(0.0, side, (3, n)) / rmax, dtype=torch.float32, device=_device())
    rr = torch.tensor(r * (rng.uniform(0.996, 1.04, n) if loose else 1.0) / rmax, dtype=torch.float32, device=_device())
    reach, box = rr[:, None] + rr[None, :], float(side / rmax)
    reach.fill_diagonal_(0.0)
    for _ in range(400):
        d = x[:, :, None] - x[:, None, :]
        d -= box * torch.round(d / box)
        dist = (d * d).sum(0).sqrt_().clamp_min_(1e-6)
        x = x + 0.35 * (d * ((reach - dist).clamp_min_(0.0) / dist)).sum(2)
    return np.mod(x.T.double().cpu().numpy() * rmax, side), r, side


def _bed(n, lo, hi, rmin, rmax, seed, which, walls, loose=False):
    """The lowest n spheres of the tiled cell that fit the container: walls(p) gives each wall's distance
    and outward direction.  A sphere that nearly reaches a wall is moved to touch it."""
    cell, cr, side = _cell(seed, rmin, rmax, loose)
    rng = _rng(seed, 2, which)
    shift = rng.uniform(0.0, side, 3)
    k = [np.arange(math.floor((lo[a] - shift[a]) / side), math.ceil((hi[a] - shift[a]) / side)) for a in range(3)]
    pos, rad = [], []
    for kz in k[2]:                      # from the bottom up, until there are enough
        t = np.stack(np.meshgrid(k[0], k[1], [kz], indexing="ij"), axis=-1).reshape(-1, 1, 3)
        p = (t * side + shift + cell[None]).reshape(-1, 3)
        r = np.broadcast_to(cr, (t.shape[0], cr.size)).ravel()
        near = np.all((p > lo) & (p < hi), axis=1)
        p, r = p[near], r[near]
        ok = np.ones(r.size, bool)
        for dist, out in walls(p):
            gap = dist - r
            ok &= gap >= 0.0
            touch = ok & (gap < 0.12 * r)
            p[touch] += ((gap + r * rng.uniform(0.0, 0.002, r.size))[:, None] * out)[touch]
        pos.append(p[ok])
        rad.append(r[ok])
        if sum(x.size for x in rad) >= n and kz * side + shift[2] > np.sort(np.concatenate([q[:, 2] for q in pos]))[n - 1]:
            break
    pos, rad = np.concatenate(pos), np.concatenate(rad)
    if rad.size < n:
        raise ValueError("the container holds %d spheres of %d" % (rad.size, n))
    low = np.argsort(pos[:, 2], kind="stable")[:n]
    pos, rad = pos[low], rad[low]
    # numbered as a bed poured from a lattice is: row by row
    row = np.floor(pos / (2.0 * rmax)).astype(np.int64)
    order = np.lexsort((row[:, 2], row[:, 1], row[:, 0]))
    return np.concatenate([pos[order], rad[order, None]], axis=1)


def _plane_walls(sc):
    def walls(p):
        for w in sc.planes:
            h = (p - w["xw"]) @ w["uw"]
            yield np.abs(h), np.where(h[:, None] < 0.0, w["uw"], -w["uw"])
    return walls


def _take(sc, pos):
    sc.pos = np.ascontiguousarray(pos)
    for k, v in scenes._state(sc.pos).items():
        setattr(sc, k, v)


def _scene(shape, n, seed, which=0, orifice=8.0, fric=0.4):
    """One scene with its state: a settled box of equal spheres, a polydisperse bed, a falling box, a
    hopper, or a drum filled to a third."""
    if shape in ("settle", "bed", "loose"):
        mono = shape == "settle"
        r = (0.005, 0.005) if mono else (0.002, 0.004)
        if mono:   # the settle's 0.3 x 0.3 x 0.5 m, its floor scaled with the count
            s = 0.5 * 0.3 * math.sqrt(n / 8000.0)
            lo, hi = np.array([-s, -s, 0.0]), np.array([s, s, 0.5])
        else:
            s = 0.5 * math.sqrt(n / 1_000_000)
            lo, hi = np.array([-s, -s, 0.0]), np.array([s, s, 2.0])
        planes, names = scenes.box_walls(lo, hi)
        cp = scenes._default_property()
        sc = scenes.Scene(name=shape, seed=seed, dt=1e-5 if mono else 5e-6, steps=0,
                          params=scenes._reference_grid(r[1], n, 1e-5 if mono else 5e-6), pos=np.zeros((1, 4)),
                          **scenes._state(np.zeros((1, 4))), cp_pp=cp, planes=planes, plane_names=names,
                          cp_planes=np.array([cp] * len(names)))
        _take(sc, _bed(n, lo, hi, *r, seed, which, _plane_walls(sc), shape == "loose"))
    elif shape == "hopper":
        sc = scenes.hopper(n=n, seed=1, orifice=orifice, fric=fric)
        v = sc.vlist.reshape(-1, 3)
        top, r_o = v[:, 2].max(), 0.5 * orifice * 0.006
        slope, half = math.tan(math.radians(60.0)), math.pi / 64
        r_top = r_o + top / slope

        def walls(p):   # the facet of the cone that a sphere lies over, and nothing below the orifice
            a = (np.floor(np.arctan2(p[:, 1], p[:, 0]) / (2 * half)) + 0.5) * 2 * half
            c = np.cos(half)
            dist = (r_o + p[:, 2] / slope) * c - (p[:, 0] * np.cos(a) + p[:, 1] * np.sin(a))
            nrm = math.hypot(1.0, c / slope)
            out = np.stack([np.cos(a), np.sin(a), np.full(a.size, -c / slope)], axis=1) / nrm
            yield np.where(p[:, 2] > 0.004, dist / nrm, -1.0), out
        _take(sc, _bed(n, np.array([-r_top, -r_top, 0.0]), np.array([r_top, r_top, top]), 0.002, 0.004, seed, which, walls))
    else:
        sc = scenes.drum_lattice(n=1000, seed=1)
        radius, half = 0.5 * math.cos(math.pi / 242), 0.2

        def walls(p):
            rho = np.maximum(np.hypot(p[:, 0], p[:, 2]), 1e-9)
            yield radius - rho, np.stack([p[:, 0] / rho, np.zeros(rho.size), p[:, 2] / rho], axis=1)
            yield half - np.abs(p[:, 1]), np.stack([np.zeros(rho.size), np.sign(p[:, 1]), np.zeros(rho.size)], axis=1)
        _take(sc, _bed(n, np.array([-0.5, -half, -0.5]), np.array([0.5, half, 0.5]), 0.002, 0.004, seed, which, walls))
    rng = _rng(seed, 4, which)
    sc.vel[:] = rng.normal(0.0, 0.02, sc.vel.shape)
    sc.omega[:] = rng.normal(0.0, 2.0, sc.omega.shape)
    sc.params["np"] = n
    return sc


def _scenes_of(case, seed):
    """Every scene of a case, in order."""
    if case["kind"] == "batch":       # hoppers as in the discharge batch: log-uniform from 2,000 to 200,000
        return [_scene("hopper", d["n"], seed, k, d["orifice"], d["fric"])
                for k, d in enumerate(scenes.hopper_batch(count=case["count"], seed=11))]
    if case["kind"] == "served":      # requests as a server gets them, at different ages: boxes falling, hoppers packed
        got = []
        for k, d in enumerate(scenes.served_requests(count=case["count"], seed=9, n_max=200_000)):
            a = d["kwargs"]
            got.append(_scene("loose", a["n"], seed, k) if d["kind"] == "box" else
                       _scene("hopper", max(a["n"], 2000), seed, k, a["orifice"], a["fric"]))
        return got
    return [_scene(case["shape"], case["n"], seed, 0, case.get("orifice", 8.0), case.get("fric", 0.4))]


# ------------------------------------------------------------------ a pass

def _flat(arrays, dtype):
    """The arrays back to back in one device tensor, and a view of each."""
    sizes = [a.size for a in arrays]
    flat = torch.from_numpy(np.concatenate([np.asarray(a, dtype).ravel() for a in arrays])).cuda()
    return flat, list(flat.split(sizes))


class _Job:
    """A scene on the device with its input and output in pinned memory."""

    def __init__(self, sc, mode):
        self.ds = engine.DeviceScene(sc, mode=mode)
        self.n = sc.np_
        names = FIELDS + (("mass", "inertia") if mode == engine.MODE_MIXED else ("force", "moment", "mass", "inertia"))
        block = torch.from_numpy(np.concatenate([getattr(sc, k).ravel() for k in names])).pin_memory()
        self.given = dict(zip(names, block.split([WIDTH[k] * self.n for k in names])))
        out = torch.empty(16 * self.n, dtype=torch.float64).pin_memory()
        self.got = {k: v.view(self.n, WIDTH[k]) for k, v in zip(FIELDS, out.split([WIDTH[k] * self.n for k in FIELDS]))}

    def upload(self):
        at = {k: v.data_ptr() for k, v in self.given.items()}
        call("xd_scene_upload_async", self.ds.handle, *[at.get(k) for k in WIDTH], 0)

    def download(self):
        call("xd_scene_download_async", self.ds.handle, *[self.got[k].data_ptr() for k in FIELDS], None, None, 0)


def prepare(case, seed):
    kind, scs = case["kind"], _scenes_of(case, seed)
    sc, s = scs[0], {"kind": kind, "steps": case.get("steps", 1)}
    if kind in ("job", "batch", "served"):
        mode = engine.MODE_FP64 if case.get("mode") == "fp64" else engine.MODE_MIXED
        s["jobs"] = [_Job(x, mode) for x in scs]
        if kind == "job" and case["shape"] == "drum":
            s["jobs"][0].ds.set_kinematic_bodies(True)
            s["pmi"] = sc.pmi
        if kind == "batch":
            s["batch"] = engine.Batch([j.ds for j in s["jobs"]])
        return s
    s["params"] = sc.params
    if kind == "float":
        s["params_f"] = to_single(sc.params.reshape(1), PARAMS_F)
        s["at_start"], s["views"] = _flat([getattr(sc, k) for k in WIDTH], np.float32)
        s["flat"] = s["at_start"].clone()
        s["state"] = {k: v.view(-1, WIDTH[k]) for k, v in zip(WIDTH, s["flat"].split([v.numel() for v in s["views"]]))}
        s["cp"] = dem.to_dev(to_single(sc.cp_pp.reshape(1), CONTACT_PROPERTY_F))
        s["planes"] = [dem.to_dev(x.reshape(1)) for x in to_single(sc.planes, PLANE_F)]
        s["cps"] = [dem.to_dev(x.reshape(1)) for x in to_single(sc.cp_planes, CONTACT_PROPERTY_F)]
        n, nc = sc.np_, int(sc.params["ncell"])
        s["grid"] = [torch.zeros(k, dtype=torch.int32, device="cuda") for k in (n, n, nc, nc, n)]
        return s
    sim = dem.DemSimulation()
    sim.initialize(sc)
    s["sim"], s["n"] = sim, sc.np_
    if kind == "step":     # the state in one tensor, so that it is set back by one copy
        names = ("dpos", "dvel", "dacc", "davel", "daacc", "dforce", "dmoment")
        s["at_start"], views = _flat([dem.from_dev(getattr(sim, k)) for k in names], np.float64)
        s["flat"] = s["at_start"].clone()
        for k, v, a in zip(names, s["flat"].split([v.numel() for v in views]), views):
            setattr(sim, k, v.view(sc.np_, -1))
    elif kind == "contacts":
        sim.dtor.detection(sim.dpos, sim.cm.SphereData(), sim.np, sim.nPolySphere)
        s["sums"] = torch.zeros(2, sc.np_, 3, dtype=torch.float64, device="cuda")
        sim.dforce, sim.dmoment = s["sums"][0], s["sums"][1]
        if sc.ntri:
            s["bodies"] = sim.cm.cppoly.dpmi.clone()
    return s


def run(s):
    kind = s["kind"]
    if kind in ("job", "batch", "served"):
        jobs = s["jobs"]
        if "pmi" in s:                        # the drum from its first pose
            jobs[0].ds.set_bodies(s["pmi"])
        for j in jobs:
            j.upload()
        if kind == "job":
            jobs[0].ds.step(s["steps"])
        elif kind == "batch":
            s["batch"].step(s["steps"])
        else:
            engine.step_many([j.ds for j in jobs], s["steps"])
        for j in jobs:
            j.download()
        out = [j.got for j in jobs]
        if "pmi" in s:                        # the pose reached and the reaction on the drum
            out.append(torch.from_numpy(jobs[0].ds.get_bodies().view(np.float64).reshape(-1, 20)))
        return out
    dem.set_symbolic_parameter(s["params"])   # the interface has one parameter block: this simulation's
    if kind == "float":
        return _float_step(s)
    sim = s["sim"]
    if kind == "grid":
        sim.dtor.detection(sim.dpos, None, sim.np, 0)
        return {k: getattr(sim.dtor, k)() for k in ("cellID", "bodyID", "sortedID", "cellStart", "cellEnd")}
    if kind == "contacts":
        s["sums"].zero_()
        if "bodies" in s:
            sim.cm.cppoly.dpmi.copy_(s["bodies"])
        sim.cm.runCollision(sim.dpos, sim.dvel, sim.davel, sim.dmass, sim.dforce, sim.dmoment, sim.dtor.sortedID(),
                            sim.dtor.cellStart(), sim.dtor.cellEnd(), sim.np)
        return [sim.dforce, sim.dmoment] + ([sim.cm.cppoly.dpmi.view(torch.float64).view(-1, 20)] if "bodies" in s else [])
    s["flat"].copy_(s["at_start"])
    sim.oneStepAnalysis()
    return {"pos": sim.dpos, "vel": sim.dvel, "acc": sim.dacc, "omega": sim.davel, "alpha": sim.daacc}


def _float_step(s):
    """One step of the single precision interface in the reference's order."""
    s["flat"].copy_(s["at_start"])
    call("xd_set_symbolic_parameter_f", s["params_f"].ctypes.data)
    st, n = {k: v.data_ptr() for k, v in s["state"].items()}, s["state"]["mass"].numel()
    h, ix, cs, ce, so = (t.data_ptr() for t in s["grid"])
    call("xd_vv_update_position_f", st["pos"], st["vel"], st["acc"], n, 0)
    call("xd_calculate_hash_and_index_f", h, ix, st["pos"], n, 0)
    call("xd_reorder_and_find_cell_start_f", h, ix, cs, ce, so, n, s["grid"][2].numel(), 0)
    args = [st[k] for k in ("pos", "vel", "omega", "force", "moment", "mass")]
    call("xd_calculate_p2p_f", 1, *args, so, cs, ce, s["cp"].data_ptr(), n, 0)
    for p, c in zip(s["planes"], s["cps"]):
        call("xd_plane_contact_force_f", 1, p.data_ptr(), *args, n, c.data_ptr(), 0)
    call("xd_vv_update_velocity_f", *[st[k] for k in ("vel", "acc", "omega", "alpha", "force", "moment", "mass", "inertia")],
         n, 0)
    return {k: s["state"][k] for k in FIELDS}


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Inputs read once and outputs written once; about 5 contacts a sphere in a bed (each pair once, some
    200 operations) and 150 operations of the integration a step."""
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "batch":
        n, packed = sum(d["n"] for d in scenes.hopper_batch(count=case["count"], seed=11)), 1.0
    elif kind == "served":
        got = [(d["kwargs"]["n"], d["kind"]) for d in scenes.served_requests(count=case["count"], seed=9, n_max=200_000)]
        n = sum(a for a, _ in got)
        packed = sum(a for a, k in got if k == "hopper") / n
    else:
        n, packed = case["n"], 0.0 if case["shape"] == "loose" else 1.0
    mesh = {"hopper": 4096, "drum": 20480}.get(case.get("shape"), 0) * 152.0
    contact, advance = 2.3 * 200.0 * packed, 150.0
    if kind == "grid":
        return {"bytes": n * (32.0 + 12.0) + 8.0 * 128 ** 3, "flops": 6.0 * n}
    if kind == "contacts":
        return {"bytes": n * 8.0 * (4 + 3 + 3 + 1 + 6) + 4.0 * n + mesh, "flops": n * contact}
    each = 4.0 if kind == "float" else 8.0
    return {"bytes": n * each * (18 + 16) + mesh, "flops": n * steps * (contact + advance)}


# ------------------------------------------------------------------ the same in 64 bits

def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_device())


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _pairs(x, r, slack):
    """Pairs i < j with a gap below `slack`, by a cell list."""
    size = 2.0 * float(r.max()) + slack
    c = torch.floor((x - x.min(0).values) / size).long() + 1
    dims = c.max(0).values + 2
    key = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
    order = torch.argsort(key, stable=True)
    sk, seen = key[order], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            k = key + (dx * dims[1] + dy) * dims[2]
            lo, hi = torch.searchsorted(sk, k - 1), torch.searchsorted(sk, k + 1, right=True)
            cnt = hi - lo
            i = torch.repeat_interleave(torch.arange(key.numel(), device=x.device), cnt)
            j = order[torch.arange(i.numel(), device=x.device) - torch.repeat_interleave(torch.cumsum(cnt, 0) - cnt, cnt) +
                      torch.repeat_interleave(lo, cnt)]
            keep = i < j
            i, j = i[keep], j[keep]
            near = (x[i] - x[j]).norm(dim=1) < (r[i] + r[j])[:, 0] + slack
            seen.append(torch.stack([i[near], j[near]]))
    return torch.cat(seen, dim=1)


def _law(cp, meq, req, depth, dv, u, dt):
    """The Hertz-Mindlin (DHS) normal and tangential force of a contact."""
    eeq = cp["Ei"] * cp["Ej"] / (cp["Ei"] * (1 - cp["prj"] ** 2) + cp["Ej"] * (1 - cp["pri"] ** 2))
    kn = (4.0 / 3.0) * eeq * req.sqrt()
    vn = (4.0 * meq * kn / (1.0 + (math.pi / math.log(cp["rest"])) ** 2)).sqrt()
    vu = _dot(dv, u)
    fn = (-kn * depth ** 1.5 + vn * vu) * u
    e = dv - vu * u
    m = e.norm(dim=-1, keepdim=True)
    sh = torch.where(m > 0, e / m.clamp_min(1e-300), torch.zeros_like(e))
    sr = cp["sratio"]
    return fn, torch.minimum(kn * sr * m * dt + vn * sr * m, cp["fric"] * fn.norm(dim=-1, keepdim=True)) * sh


def _closest(a, b, c, p):
    """The closest point of triangle abc to p (Ericson, Real-Time Collision Detection, 5.1.5)."""
    ab, ac = b - a, c - a
    d1, d2 = _dot(ab, p - a), _dot(ac, p - a)
    d3, d4 = _dot(ab, p - b), _dot(ac, p - b)
    d5, d6 = _dot(ab, p - c), _dot(ac, p - c)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    s = va + vb + vc
    q = a + vb / s * ab + vc / s * ac
    w = (d4 - d3) / ((d4 - d3) + (d5 - d6))
    q = torch.where((va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0), b + w * (c - b), q)
    q = torch.where((vb <= 0) & (d2 >= 0) & (d6 <= 0), a + d2 / (d2 - d6) * ac, q)
    q = torch.where((d6 >= 0) & (d5 <= d6), c, q)
    q = torch.where((vc <= 0) & (d1 >= 0) & (d3 <= 0), a + d1 / (d1 - d3) * ab, q)
    q = torch.where((d3 >= 0) & (d4 <= d3), b, q)
    return torch.where((d1 <= 0) & (d2 <= 0), a, q)


class _Exact:
    """A scene in 64 bits with plain torch: pairs, walls (their faces, all that these beds touch) and triangles."""

    def __init__(self, sc, single=False):
        one = (lambda a: np.asarray(a, np.float32).astype(np.float64)) if single else np.asarray
        rec = lambda c: {k: float(one(c[k])) for k in c.dtype.names}  # noqa: E731
        self.x, self.r = _t(one(sc.pos[:, :3])), _t(one(sc.pos[:, 3:4]))
        self.v, self.a, self.w, self.al = (_t(one(getattr(sc, k))) for k in ("vel", "acc", "omega", "alpha"))
        self.m, self.inertia = _t(one(sc.mass))[:, None], _t(one(sc.inertia))[:, None]
        self.dt, self.h2 = float(one(sc.params["dt"])), float(one(sc.params["half2dt"]))
        self.g, self.cp = _t(one(sc.params["gravity"])), rec(sc.cp_pp)
        self.planes = [({k: _t(one(p[k])) for k in ("xw", "uw")}, rec(c)) for p, c in zip(sc.planes, sc.cp_planes)]
        self.slack = 1e-3
        self.ij = _pairs(self.x, self.r, self.slack)
        self.tri, self.turned = None, 0.0
        if sc.ntri:
            self.tri, self.cpb = _t(sc.vlist.reshape(-1, 3, 3)), rec(sc.cp_poly[0])
            self.spin, self.bvel = _t(sc.pmi["omega"][0]), _t(sc.pmi["vel"][0])
            mid, rad = _t(sc.sphere[:, :3]).float(), _t(sc.sphere[:, 3]).float()
            near = []
            for k in range(0, self.x.shape[0], 50_000):
                xk = self.x[k:k + 50_000].float()
                d = torch.cdist(xk, mid, compute_mode="donot_use_mm_for_euclid_dist")
                i, t = torch.nonzero(d < rad[None, :] + self.r[k:k + 50_000].float() + 2e-3, as_tuple=True)
                near.append(torch.stack([i + k, t]))
            self.it = torch.cat(near, dim=1)
            q = _closest(*self.tri[self.it[1]].unbind(1), self.x[self.it[0]])
            self.it = self.it[:, (self.x[self.it[0]] - q).norm(dim=1) < self.r[self.it[0], 0] + 2e-3]
        self.react = torch.zeros(6, dtype=torch.float64, device=self.x.device)

    def contacts(self):
        F, M = torch.zeros_like(self.x), torch.zeros_like(self.x)
        i, j = self.ij
        d = self.x[j] - self.x[i]
        dist = d.norm(dim=1, keepdim=True)
        hit = (self.r[i] + self.r[j] - dist)[:, 0] > 0
        i, j, d, dist = i[hit], j[hit], d[hit], dist[hit]
        ri, rj, mi, mj, u = self.r[i], self.r[j], self.m[i], self.m[j], d / dist
        rv = (self.v[j] - torch.cross(self.w[j], rj * u, dim=1)) - (self.v[i] + torch.cross(self.w[i], ri * u, dim=1))
        fn, ft = _law(self.cp, mi * mj / (mi + mj), ri * rj / (ri + rj), ri + rj - dist, rv, u, self.dt)
        F.index_add_(0, i, fn + ft).index_add_(0, j, -(fn + ft))
        M.index_add_(0, i, torch.cross(ri * u, ft, dim=1)).index_add_(0, j, torch.cross(rj * u, ft, dim=1))
        for p, cp in self.planes:
            n = p["uw"] / p["uw"].norm()
            h = _dot(self.x - p["xw"], n)
            k = torch.nonzero((self.r - h.abs())[:, 0] > 0)[:, 0]
            u = torch.where(h[k] < 0, n, -n)
            fn, ft = _law(cp, self.m[k], self.r[k], self.r[k] - h[k].abs(),
                          -(self.v[k] + torch.cross(self.w[k], self.r[k] * u, dim=1)), u, self.dt)
            F.index_add_(0, k, fn + ft)
        if self.tri is not None:
            c, s = math.cos(self.turned), math.sin(self.turned)   # a body turns about y
            turn = torch.tensor([[c, 0, s], [0, 1, 0], [-s, 0, c]], dtype=torch.float64, device=self.x.device)
            i, t = self.it
            a, b, e = (self.tri[t] @ turn.T).unbind(1)
            q = _closest(a, b, e, self.x[i])
            depth = self.r[i] - (self.x[i] - q).norm(dim=1, keepdim=True)
            hit = depth[:, 0] > 0
            i, a, b, e, q, depth = i[hit], a[hit], b[hit], e[hit], q[hit], depth[hit]
            u = -torch.cross(b - a, e - a, dim=1)
            u = u / u.norm(dim=1, keepdim=True)
            dv = self.bvel + torch.cross(self.spin.expand_as(q), q, dim=1) - (self.v[i] + torch.cross(self.w[i], self.r[i] * u, dim=1))
            fn, ft = _law(self.cpb, self.m[i], self.r[i], depth, dv, u, self.dt)
            F.index_add_(0, i, fn + ft)
            self.react -= torch.cat([(fn + ft).sum(0), torch.cross(q, fn + ft, dim=1).sum(0)])
        return F, M

    def step(self, steps):
        for _ in range(steps):
            self.turned += 0.0 if self.tri is None else float(self.spin[1]) * self.dt
            self.x = self.x + self.dt * self.v + self.h2 * self.a
            F, M = self.contacts()
            a, al = F / self.m + self.g, M / self.inertia
            self.v, self.w = self.v + 0.5 * self.dt * (self.a + a), self.w + 0.5 * self.dt * (self.al + al)
            self.a, self.al = a, al
        return dict(pos=torch.cat([self.x, self.r], 1), vel=self.v, acc=self.a, omega=self.w, alpha=self.al)


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":
        return None      # whole numbers
    scs = _scenes_of(case, seed)
    if kind == "contacts":
        e = _Exact(scs[0])
        F, M = e.contacts()
        return [F, M] + ([torch.cat([_t(scs[0].pmi.view(np.float64).reshape(-1, 20))[0, :14], e.react])[None]]
                         if scs[0].ntri else [])
    if kind in ("step", "float"):
        return _Exact(scs[0], single=kind == "float").step(1)
    out = [_Exact(sc).step(case["steps"]) for sc in scs]
    return out + ([None] if case.get("shape") == "drum" else [])
