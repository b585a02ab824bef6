"""Performance cases of the DEM step: what a host program asks of this library, from its inputs in
(pinned) host memory to the state back in host memory.

Every pass of a stepping case starts from the same state, as a host program does when it hands the
library a state to advance: `update` (positions, orientations, velocities), `initialize_leapfrog`
(forces of the start state), `step(n)`, `download`.  The other cases call the per-phase entry points
in the order of the reference's time loop, the fluid coupling's step, or the differentiable run.

The states are made here, from the seed alone: packings by overlap relaxation, lattices by
pacific_b200.scenarios.  Overlaps, coordination (about 5) and density (about 0.6) are those of a settled
bed.  The passes are short because granular dynamics is chaotic: rounding differences
grow tenfold every 10 to 20 steps of a dense packing.
"""
import math

import numpy as np
import torch

import pacific_b200
from pacific_b200 import abi, scenarios

MM = 1.0e-3
RHO = 2500.0
CRUST = 0.05 * MM
F64 = torch.float64


# ---- the cases -----------------------------------------------------------------
def listed():
    return [
        # a small calibration run (1,000 spheres, one context): launch latency is all there is
        dict(name="bed 1k fp64", kind="bed", n=1000, precision="fp64", steps=101, law="hooke_memory"),
        # an ordinary single-system study; 27,000 is a full 30^3 packing
        dict(name="bed 27k mixed", kind="bed", n=27000, precision="mixed", steps=33, law="hooke_memory"),
        # the settled bed of the 200,000-sphere workload, both precisions
        dict(name="bed 200k mixed", kind="bed", n=200000, precision="mixed", steps=25, law="hooke_memory"),
        dict(name="bed 200k fp64", kind="bed", n=200000, precision="fp64", steps=25, law="hooke_memory"),
        # the same workload from its lattice: spheres falling, hardly a contact
        dict(name="fall 200k mixed", kind="fall", n=200000, precision="mixed", steps=100, law="hooke_memory"),
        # parameter studies: many independent boxes of 200 to 20,000 spheres in one context
        dict(name="ensemble 96 mixed", kind="ensemble", n=96, precision="mixed", steps=100, law="hooke_memory"),
        # cubes, cylinders and octahedra in a rotating drum
        dict(name="drum 40k mixed", kind="drum", n=40000, precision="mixed", steps=10, gjk="johnson", history=False),
        # a small box of convex bodies with the GJK warm start; the signed-volume GJK on a larger one
        dict(name="convex 2k fp64 history", kind="convex", n=2000, precision="fp64", steps=33, gjk="johnson",
             history=True),
        dict(name="convex 11k mixed sv", kind="convex", n=11111, precision="mixed", steps=17, gjk="sv", history=False),
        # the library as the collision App of a host's time loop: one call per phase and step, double precision
        dict(name="app 8k fp64", kind="app", n=8000, precision="fp64", steps=10, law="hooke_memory"),
        # immersed spheres: the fluid solver's forces in, its sub-steps, the velocities out
        dict(name="fluid 12k mixed", kind="fluid", n=12345, precision="mixed", steps=20, law="hooke_memory"),
        # calibration by gradients: run and adjoint of the 4,096-sphere workload
        dict(name="adjoint 4k fp64", kind="adjoint", n=4096, precision="fp64", steps=150),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bed", "bed", "fall", "ensemble", "drum", "convex", "app", "fluid", "adjoint"])
    c = dict(kind=kind, precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind in ("bed", "fall", "app", "fluid"):
        c["law"] = rng.choice(["hooke_memory", "hooke_memory", "hooke", "hertz_memory"])
    if kind == "bed":
        c.update(n=_size(rng, 500, 180000), steps=rng.randint(10, 33))
    elif kind == "fall":
        c.update(n=_size(rng, 1000, 200000), steps=rng.randint(30, 90))
    elif kind == "ensemble":
        c.update(n=_size(rng, 2, 90), steps=rng.randint(33, 90), law="hooke_memory")
    elif kind == "drum":
        c.update(n=_size(rng, 2000, 36000), steps=rng.randint(4, 10), gjk="johnson", history=rng.random() < 0.3)
    elif kind == "convex":
        c.update(n=_size(rng, 200, 20000), steps=rng.randint(5, 17), gjk=rng.choice(["johnson", "johnson", "sv"]),
                 history=rng.random() < 0.4)
    elif kind in ("app", "fluid"):
        c.update(n=_size(rng, 500, 50000), steps=rng.randint(5, 20))
    else:
        c.update(n=_size(rng, 200, 4096), steps=rng.randint(20, 60))
    return c


# ---- packings --------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _neighbours(x, cut, width):
    """(n, width) partners closer than `cut`, -1 where there are fewer."""
    n, dev = len(x), x.device
    lo = x.amin(0)
    dims = ((x.amax(0) - lo) / cut).floor().long() + 1
    c = ((x - lo) / cut).floor().long().minimum(dims - 1)
    key = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
    order = torch.argsort(key, stable=True)
    count = torch.bincount(key, minlength=int(dims.prod()))
    start = count.cumsum(0) - count
    most = int(count.max())
    out = torch.full((n, width + 1), -1, dtype=torch.long, device=dev)
    filled = torch.zeros(n, dtype=torch.long, device=dev)
    me = torch.arange(n, device=dev)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                d = c + torch.tensor([dx, dy, dz], device=dev)
                ok = ((d >= 0) & (d < dims)).all(1)
                k = torch.where(ok, (d[:, 0] * dims[1] + d[:, 1]) * dims[2] + d[:, 2], 0)
                for s in range(most):
                    has = ok & (s < count[k])
                    j = order[torch.where(has, start[k] + s, 0)]
                    has = has & (j != me) & (((x[j] - x) ** 2).sum(1) < cut * cut)
                    out[me, torch.where(has, filled.clamp(max=width), width)] = j
                    filled = filled + has
    if int(filled.max()) > width:
        raise ValueError("more than %d neighbours" % width)
    return torch.where(torch.arange(width, device=dev) < filled[:, None], out[:, :width], -1)


def _relax(x, cut, reach, keep, iterations, width, rebuild=25):
    """Pushes overlapping bodies apart (gradient steps with momentum).  reach(j, u): the distance at
    which body i and its partners j touch along the unit vectors u; keep(x): x inside its container."""
    v = torch.zeros_like(x)
    for k in range(iterations):
        if k % rebuild == 0:
            near = _neighbours(x, cut, width)
            ok, j = near >= 0, near.clamp(min=0)
        d = x[:, None] - x[j]
        length = d.norm(dim=2).clamp(min=1.0e-9)
        u = d / length[..., None]
        push = torch.where(ok, (reach(j, u) - length).clamp(min=0), 0.0)
        y = keep(x + 0.75 * v + 0.25 * (u * push[..., None]).sum(1))
        v, x = y - x, y
    return x


def _grid(n, shape, spacing):
    k = torch.arange(n)
    return spacing * (torch.stack([k % shape[0], k // shape[0] % shape[1], k // (shape[0] * shape[1])], 1).to(F64) + 0.5)


def _packed_spheres(n, seed):
    """Radii, centres and box size (mm) of a dense packing of spheres, r in [0.8, 1.2], in a closed box."""
    g = torch.Generator().manual_seed(seed)
    r = 0.8 + 0.4 * torch.rand(n, generator=g, dtype=F64)
    volume = float((4.0 / 3.0 * math.pi * r ** 3).sum()) / 0.6
    w = (volume / 1.5) ** (1.0 / 3.0)
    size = torch.tensor([w, w, 1.5 * w], dtype=F64)
    spacing = (volume / n) ** (1.0 / 3.0)
    m = max(1, math.ceil(w / spacing))
    x = _grid(n, (m, m), 1.0)
    top = float(x[:, 2].max()) + 0.5
    x = x * torch.tensor([w / m, w / m, 1.5 * w / top], dtype=F64) + 0.3 * (torch.rand(n, 3, generator=g, dtype=F64) - 0.5)
    dev = _device()
    x, r, size = x.to(dev), r.to(dev), size.to(dev)
    x = _relax(x, 2.4 * 1.08, lambda j, u: r[:, None] + r[j],
               lambda y: torch.minimum(torch.maximum(y, r[:, None]), size - r[:, None]), 400, 32)
    # no overlap above 0.04 mm (the crusts of a pair are 0.1 mm)
    near = _neighbours(x, 2.4, 32)
    j = near.clamp(min=0)
    length = torch.where(near >= 0, (x[:, None] - x[j]).norm(dim=2), 99.0)
    for _ in range(20):
        r = r - 0.5 * (r[:, None] + r[j] - length - 0.039).clamp(min=0).amax(1)
    return r.cpu().numpy(), x.cpu().numpy(), size.cpu().numpy()


def _packed_convex(n, seed, radius=None):
    """Shape kinds, orientations and centres (mm) of a dense packing of the cubes, cylinders and octahedra of
    scenarios.CONVEX_SHAPES: along their centre line two bodies pass each other by a few percent of their reach at
    most, so that few corners meet and the overlaps stay below the crusts.  In a
    closed box (returns its size) or, with `radius`, in a cylinder about z (returns its length)."""
    rng = np.random.default_rng(seed)
    wanted, n = n, n + n // 12 + 8  # some are left out in the end
    kinds = rng.choice(3, size=n, p=scenarios.CONVEX_FRACTIONS)
    q = scenarios.random_quaternions(n, rng)
    basis = scenarios.quaternion_basis(q).reshape(n, 3, 3)
    circ = np.array([scenarios.circumscribed_radius(t, p) for t, p in scenarios.CONVEX_SHAPES]) / MM
    volume = n * 16.3
    if radius is None:
        w = volume ** (1.0 / 3.0) + 1.0  # the bounding spheres stay inside: the outermost 0.5 mm is thinly filled
        size = np.array([w, w, w])
    else:
        size = np.array([math.sqrt(math.pi) * radius, math.sqrt(math.pi) * radius,
                         volume / (math.pi * (radius - 0.5) ** 2) + 1.0])
    spacing = (volume / n) ** (1.0 / 3.0)
    m = [max(1, math.ceil(size[a] / spacing)) for a in (0, 1)]
    x = _grid(n, m, 1.0).numpy()
    x = x * np.array([size[0] / m[0], size[1] / m[1], size[2] / (x[:, 2].max() + 0.5)])
    x = x + 0.3 * rng.uniform(-1.0, 1.0, size=(n, 3))
    if radius is not None:  # the square cross-section mapped on the disc
        p = (x[:, :2] / size[:2] * 2.0 - 1.0).clip(-0.999, 0.999)
        x[:, 0] = radius * p[:, 0] * np.sqrt(1.0 - 0.5 * p[:, 1] ** 2)
        x[:, 1] = radius * p[:, 1] * np.sqrt(1.0 - 0.5 * p[:, 0] ** 2)
    dev = _device()
    kt, bt = torch.from_numpy(kinds).to(dev), torch.from_numpy(basis).to(dev)
    ct = torch.from_numpy(circ[kinds]).to(dev)
    st = torch.from_numpy(size).to(dev)

    def support(k, b, u):
        local = torch.einsum("nkij,nki->nkj", b, u).abs()
        box = local.sum(2)
        cylinder = (local[..., 0] ** 2 + local[..., 2] ** 2).sqrt() + local[..., 1]
        return torch.where(k == 0, box, torch.where(k == 1, cylinder, 1.2 * local.amax(2)))

    def reach(j, u):
        own = support(kt[:, None].expand(j.shape), bt[:, None].expand(*j.shape, 3, 3), u)
        return 0.97 * (own + support(kt[j], bt[j], u))

    def keep(y):
        if radius is None:
            return torch.minimum(torch.maximum(y, ct[:, None]), st - ct[:, None])
        z = torch.minimum(torch.maximum(y[:, 2], ct), st[2] - ct)
        s = (((radius - ct) / y[:, :2].norm(dim=1).clamp(min=1.0e-9)).clamp(max=1.0))[:, None]
        return torch.cat([y[:, :2] * s, z[:, None]], 1)

    t = _relax(keep(torch.from_numpy(x).to(dev)), 3.6, reach, keep, 60, 48)
    t = _relax(t, 3.6, lambda j, u: reach(j, u) - 0.02, keep, 140, 48)
    near = _neighbours(t, 3.6, 48)
    j = near.clamp(min=0)
    d = t[:, None] - t[j]
    length = d.norm(dim=2).clamp(min=1.0e-9)
    close = (reach(j, d / length[..., None]) - length).masked_fill(near <= torch.arange(n, device=dev)[:, None], -1.0)
    # the bodies closest to another one are left out
    own = torch.argsort(close.amax(1), stable=True)[:wanted].sort().values.cpu().numpy()
    return kinds[own], q[own], basis.reshape(n, 9)[own], t.cpu().numpy()[own], size


# ---- scenarios -------------------------------------------------------------------
LAWS = {
    "hooke_memory": (abi.HOOKE_MEMORY, [1.0e5, 0.9, -1.0, 0.5, 0.8e5, 0.0, 0.0, 0.0]),
    "hooke": (abi.HOOKE, [1.0e5, 0.9, -1.0, 0.5, 0.0]),
    "hertz_memory": (abi.HERTZ_MEMORY, [2.0e8, 0.9, 0.5, 6.0e7, 0.0, 0.0, 0.0]),
}


def _spheres(r, x, v, w):
    n = len(r)
    q = np.zeros((n, 4))
    q[:, 3] = 1.0
    return dict(id=np.arange(n, dtype=np.int32), system=None, shape=np.zeros(n, np.int32),
                material=np.zeros(n, np.int32), radius=r, crust=np.full(n, CRUST), mass=RHO * 4.0 / 3.0 * math.pi * r ** 3,
                inertia=np.repeat((RHO * 8.0 / 15.0 * math.pi * r ** 5)[:, None], 3, 1), position=x, quaternion=q,
                basis=None, velocity=v, omega=w)


def _boxed(name, particles, lo, hi, law, cell, faces="xXyYzZ", dt=5.0e-6, shapes=None):
    shapes = list(shapes or [(abi.SPHERE, [1.0 * MM])])
    walls, obstacles = scenarios.box_walls(lo, hi, faces, 0.5 * MM, CRUST, len(shapes), -1)
    laws = [[(0, 0, *law), (0, 1, *law)]]
    domain = [dict(origin=lo, size=hi - lo, cell_size=cell, gravity=(0.0, 0.0, -9.81))]
    return scenarios.Scenario(name, shapes + walls, domain, laws, [obstacles], particles, dt, 0)


def _scenario(case, seed):
    kind, n = case["kind"], case["n"]
    rng = np.random.default_rng(seed)
    if kind in ("bed", "app", "fluid"):
        r, x, size = _packed_spheres(n, seed)
        p = _spheres(r * MM, x * MM, rng.normal(0.0, 0.01, (n, 3)), rng.normal(0.0, 5.0, (n, 3)))
        # the walls reach 1 um into the outermost spheres
        # (the added inertia of immersed spheres is negative here, 1 - 1000 / 2500: they need a smaller step)
        return _boxed("bed", p, np.full(3, 0.001 * MM), (size - 0.001) * MM, LAWS[case["law"]], 2.4 * MM,
                      dt=2.0e-6 if kind == "fluid" else 5.0e-6)
    if kind == "fall":
        m = max(2, round((n / 3.6) ** (1.0 / 3.0)))  # 38 x 38 for 200,000, as in that workload
        lo, hi = np.zeros(3), np.array([m, m, math.ceil(n / (m * m)) + 2]) * 2.6 * MM
        x = scenarios.lattice(n, lo, hi, 2.6 * MM, 1.3 * MM, 0.1 * MM, rng)
        p = _spheres(rng.uniform(0.8 * MM, 1.2 * MM, n), x, rng.normal(0.0, 0.05, (n, 3)), np.zeros((n, 3)))
        return _boxed("fall", p, lo, hi, LAWS[case["law"]], 2.4 * MM, faces="xXyYz")
    if kind == "ensemble":
        sc = scenarios.ensemble_512(n_systems=n)  # sizes and laws of that workload's first systems
        m = sc.n
        sc.particles["position"] = sc.particles["position"] + rng.uniform(-0.03 * MM, 0.03 * MM, (m, 3))
        sc.particles["velocity"] = rng.normal(0.0, 0.3, (m, 3))
        sc.particles["omega"] = rng.normal(0.0, 5.0, (m, 3))
        return sc
    if kind == "adjoint":
        return scenarios.adjoint_4k(seed=seed, vseed=seed + 1, n=n)
    radius = None if kind == "convex" else 0.85 * (n * 16.3) ** (1.0 / 3.0)
    kinds, q, basis, x, size = _packed_convex(n, seed, radius)
    p = scenarios._convex_particles(x * MM, np.random.default_rng(0), crust=CRUST)
    for k, (t, prm) in enumerate(scenarios.CONVEX_SHAPES):
        volume, inertia = scenarios.shape_volume_inertia(t, prm)
        own = kinds == k
        p["mass"][own], p["inertia"][own] = RHO * volume, RHO * inertia
        p["radius"][own] = scenarios.circumscribed_radius(t, prm)
    p.update(shape=kinds.astype(np.int32), quaternion=q, basis=basis, velocity=rng.normal(0.0, 0.05, (n, 3)),
             omega=rng.normal(0.0, 20.0, (n, 3)))
    law = (abi.HOOKE_MEMORY, [2.0e5, 0.7, -1.0, 0.4, 1.6e5, 0.0, 0.0, 0.0])
    circ = float(p["radius"].max())
    if kind == "convex":
        sc = _boxed("convex", p, np.zeros(3), size * MM, law, 2.0 * circ, dt=2.0e-6, shapes=scenarios.CONVEX_SHAPES)
    else:
        # the drum's lattice fill is replaced by the packing; its shell boxes reach 0.02 mm inwards
        sc = scenarios.drum(n=1, radius=(radius - 0.02) * MM, length=(size[2] - 0.02) * MM)
        p["position"][:, 2] -= 0.01 * MM
        sc.particles = p
    return sc


# ---- state, pass -----------------------------------------------------------------
class _State:
    pass


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def prepare(case, seed):
    s = _State()
    s.case, s.sc = case, _scenario(case, seed)
    sc = s.sc
    if case.get("gjk") == "sv":
        sc.meta["collision"] = abi.GJK_SV
    if case.get("history"):
        sc.meta["collision_options"] = dict(history=True)
    s.sim = abi.Simulation(pacific_b200.load_library(), abi.MIXED if case["precision"] == "mixed" else abi.FP64,
                           max_particles=sc.n, n_systems=len(sc.domains))
    scenarios.apply(s.sim, sc)
    n = sc.n
    keys = ["position", "quaternion", "velocity", "omega"] + (["basis"] if sc.particles["basis"] is not None else [])
    s.start = {k: _pinned(sc.particles[k]) for k in keys}
    widths = dict(position=3, quaternion=4, velocity=3, omega=3, force=3, torque=3)
    s.out = {k: _pinned(np.zeros((n, w))) for k, w in widths.items()}
    s.out["coordination"] = _pinned(np.zeros(n, np.int32))
    rng = np.random.default_rng(seed + 7)
    if case["kind"] == "fluid":
        weight = float(sc.particles["mass"].mean()) * 9.81
        s.hydro = (_pinned(rng.normal(0.0, 0.3 * weight, (n, 3))), _pinned(rng.normal(0.0, 0.1 * weight * MM, (n, 3))))
        s.sim.set_fluid(1000.0, True, np.full(n, RHO))
    if case["kind"] == "adjoint":
        s.adjoint = abi.Adjoint(s.sim, checkpoint_every=50)
        s.cotangents = tuple(rng.normal(0.0, 1.0, (n, 3)) for _ in range(3))
    return s


def run(s):
    sim, steps, dt, kind = s.sim, s.case["steps"], s.sc.dt, s.case["kind"]
    if kind == "adjoint":
        final = s.adjoint.forward(steps, dt)
        grads = s.adjoint.backward(*s.cotangents)
        return {"final": final, "gradient": grads}
    sim.update(s.start)
    if kind == "app":
        sim.link_update()
        sim.initialize_leapfrog(0.0, dt)
        for k in range(steps):
            sim.move(k * dt, 0.5 * dt, dt)
            sim.link_update(k * dt, dt)
            sim.compute_forces(k * dt, dt)
            sim.advance_velocity(k * dt, 0.5 * dt)
    elif kind == "fluid":
        sim.set_hydro_forces(*s.hydro)
        sim.initialize_leapfrog(0.0, dt)
        sim.fluid_step((steps + 0.5) * dt, dt, dt, 1, 0.0)
    else:
        sim.initialize_leapfrog(0.0, dt)
        sim.step(steps, 0.0, dt)
    return sim.download(s.out)


# ---- work and tolerance -----------------------------------------------------------
def _particles(case):
    # the ensemble's sizes are log-uniform in [200, 20000]: 4,300 on average
    return case["n"] * 4300 if case["kind"] == "ensemble" else case["n"]


def work(case):
    n, mixed = _particles(case), case["precision"] == "mixed"
    z = dict(bed=5.2, app=5.2, fluid=5.2, fall=0.01, ensemble=0.5, drum=2.0, convex=2.0, adjoint=1.0)[case["kind"]]
    # a step reads and writes each particle's state once, and each contact's memory once
    per_step = n * ((247.0 if mixed else 355.0) + (44.0 if mixed else 80.0) * z)
    if case["kind"] in ("drum", "convex"):
        per_step += n * 144.0  # the basis
    per_step *= case["steps"]
    flops = n * case["steps"] * (300.0 + 0.5 * z * 400.0)
    if case["kind"] in ("drum", "convex"):
        flops += n * case["steps"] * 3.5 * 10.0 * 300.0  # 3.5 GJK runs of 10 iterations a body
    if case["kind"] == "adjoint":
        return {"bytes": 3.0 * per_step + n * 8.0 * 27.0, "flops": 4.0 * flops}
    return {"bytes": per_step + n * 8.0 * 32.0, "flops": flops}


def tolerance(case):
    """About four times what another order of the force sums (cells 1.25 times as wide) changes, and what the 64-bit
    restatement differs by, over the steps of the cases: rounding that the dynamics has amplified."""
    convex, mixed = case["kind"] in ("drum", "convex"), case["precision"] == "mixed"
    if convex:  # contact points on flat faces hinge on the last bits of the poses
        return {"rel": 2.0e-2, "max": 0.9, "differ": 1.0e-3} if mixed else {"rel": 5.0e-4, "max": 3.0e-2, "differ": 1.0e-3}
    if mixed:
        return {"rel": 1.0e-2, "max": 0.9, "differ": 1.0e-3}
    return {"rel": 1.0e-8, "max": 1.0e-6, "differ": 1.0e-5}


# ---- the same runs in 64 bits, in torch --------------------------------------------
def _norm(a):
    s = (a * a).sum(-1)
    return torch.where(s > 0, s, 1.0).sqrt() * (s > 0)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(a):
    s = (a * a).sum(-1, keepdim=True)
    return a / torch.where(s > 0, s, 1.0).sqrt()


def _hooke_memory(pen, v0, w0, l0, v1, w1, l1, m0, m1, p, dt, kd, pn, existed):
    """Force on the first body of every contact of the HookeMemory law, and the new memory."""
    kn, en, muc, kt = p
    beta = en.log() / (math.pi ** 2 + en.log() ** 2).sqrt()
    normal = _unit(pen)
    rel = v0 + _cross(w0, l0) - v1 - _cross(w1, l1)
    vn = normal * _dot(rel, normal)
    vt = rel - vn
    m = 1.0 / (1.0 / m0 + 1.0 / m1)
    fn = pen * kn + 2.0 * beta * (m * kn).sqrt() * vn
    nfn = _norm(fn)[..., None]
    gammat = -2.0 * beta * (kn / m).sqrt() * m
    # the spring turned by the rotation from the last normal to this one
    qv, qw = _cross(pn, normal), 1.0 + _dot(pn, normal)
    s = (qv * qv).sum(-1, keepdim=True) + qw * qw
    s = torch.where(s > 0, s, 1.0).sqrt()
    qv, qw = qv / s, qw / s
    turned = kd * (qw * qw - _dot(qv, qv)) + 2.0 * qv * _dot(kd, qv) + 2.0 * qw * _cross(qv, kd)
    kd = torch.where(existed, turned, 0.0) + vt * (dt * kt)
    nvt = _norm(vt)[..., None]
    t = torch.where(nvt > 1.0e-3, -_unit(vt), -_unit(kd + vt * gammat))
    nft = _norm(kd + gammat * vt)[..., None]
    slip = nft > muc * nfn
    ft = t * torch.where(slip, muc * nfn, nft)
    kd = torch.where(slip, (-t * muc * nfn - gammat * vt) / kt, kd)
    return fn + ft, kd, normal


def _leapfrog(sc, steps, dt, params, box, x, v, w, reach, fluid=None):
    """The leapfrog of spheres in closed or open boxes.  params(k): law parameters of sphere pairs (0) and
    walls (1) per contact row; box: per sphere the faces (n, 3) low, high and which of them are there (n, 6);
    reach: pairs that start further apart do not meet."""
    dev = x.device
    p = sc.particles
    r, m, inertia = (torch.from_numpy(np.ascontiguousarray(a)).to(dev)[:, None] for a in
                     (p["radius"], p["mass"], p["inertia"][:, 0]))
    cut = 2.0 * float(r.max()) + reach
    system = p.get("system")
    apart = torch.zeros_like(x)
    if system is not None:  # systems do not meet
        apart[:, 0] = torch.from_numpy(np.asarray(system)).to(dev).to(F64)
    near = _neighbours((x + apart).detach(), cut, 40)
    i, k = (near > torch.arange(len(x), device=dev)[:, None]).nonzero(as_tuple=True)
    j = near[i, k]
    low, high, there = box
    gravity = torch.tensor(sc.domains[0]["gravity"], dtype=F64, device=dev)
    pair, wall = params(i, 0), params(torch.arange(len(x), device=dev), 1)
    big, zero = torch.full_like(m, 1.0e20), torch.zeros_like(x)
    cf = 1.0 - fluid[0] if fluid else 1.0
    memory = [(torch.zeros(len(i), 3, dtype=F64, device=dev),) * 2 + (torch.zeros(len(i), 1, dtype=bool, device=dev),)]
    memory += [(zero, zero, torch.zeros(len(x), 1, dtype=bool, device=dev)) for _ in range(6)]

    def forces(x, v, w, memory, dt):
        out = []
        f, t = m * gravity * cf, torch.zeros_like(x)
        ab = x[j] - x[i]
        length = _norm(ab)[:, None]
        gap = length - (r[i] + r[j])
        touch = gap < 0
        u = ab / length
        point = u * (r[i] + 0.5 * gap)
        fij, kd, nn = _hooke_memory(torch.where(touch, u * gap, u), v[i], w[i], point, v[j], w[j], point - ab, m[i], m[j],
                                    pair, dt, *memory[0])
        fij = torch.where(touch, fij, 0.0)
        out.append((torch.where(touch, kd, 0.0), nn, touch))
        f = f.index_add(0, i, fij).index_add(0, j, -fij)
        t = t.index_add(0, i, _cross(point, fij)).index_add(0, j, -_cross(point - ab, fij))
        count = torch.zeros(len(x), dtype=torch.long, device=dev).index_add(0, i, touch[:, 0].long())
        count = count.index_add(0, j, touch[:, 0].long())
        for face in range(6):
            axis, sign = face // 2, (-1.0 if face % 2 == 0 else 1.0)
            u = torch.zeros(3, dtype=F64, device=dev)
            u[axis] = sign
            at = (low if face % 2 == 0 else high)[:, axis:axis + 1]
            gap = sign * (at - x[:, axis:axis + 1]) - r
            touch = (gap < 0) & there[:, face:face + 1]
            lever = u * (r + 0.5 * gap)
            fw, kd, nn = _hooke_memory(torch.where(touch, u * gap, u), v, w, lever, zero, zero, lever, m, big, wall, dt,
                                       *memory[1 + face])
            fw = torch.where(touch, fw, 0.0)
            out.append((torch.where(touch, kd, 0.0), nn, touch))
            f, t, count = f + fw, t + _cross(lever, fw), count + touch[:, 0]
        if fluid:
            f, t = f + fluid[1], t + fluid[2]
        return f, t, out, count

    q = torch.from_numpy(p["quaternion"]).to(dev)
    f, t, memory, count = forces(x, v, w, memory, sc.dt)  # initialize_leapfrog
    memory = [(torch.zeros_like(a), b, c) for a, b, c in memory]
    for _ in range(steps):
        v = v + f / (m * cf) * (0.5 * dt)
        w = w + t / (inertia * cf) * (0.5 * dt)
        x = x + v * dt
        with torch.no_grad():
            nw = _norm(w)[:, None]
            dq = torch.cat([_unit(w) * (0.5 * dt * nw).sin(), (0.5 * dt * nw).cos()], 1)
            q = torch.cat([_cross(dq[:, :3], q[:, :3]) + dq[:, 3:] * q[:, :3] + q[:, 3:] * dq[:, :3],
                           dq[:, 3:] * q[:, 3:] - _dot(dq[:, :3], q[:, :3])], 1)
        f, t, memory, count = forces(x, v, w, memory, dt)
        v = v + f / (m * cf) * (0.5 * dt)
        w = w + t / (inertia * cf) * (0.5 * dt)
    return dict(position=x, quaternion=q, velocity=v, omega=w, force=f, torque=t, coordination=count)


def exact(case, seed):
    kind = case["kind"]
    # convex bodies: a contact's points are not unique on flat faces, and 64-bit distances of every pair
    # take minutes in torch; the other laws have no restatement here
    if kind in ("drum", "convex") or case.get("law", "hooke_memory") != "hooke_memory":
        return None
    sc, dev = _scenario(case, seed), _device()
    p, n = sc.particles, sc.n
    system = np.zeros(n, int) if p.get("system") is None else np.asarray(p["system"])
    low = np.stack([np.asarray(d["origin"], float) for d in sc.domains])
    high = low + np.stack([np.asarray(d["size"], float) for d in sc.domains])
    faces = "xXyYzZ" if kind not in ("fall", "adjoint") else "xXyYz"
    there = np.tile(np.array([f in faces for f in "xXyYzZ"]), (n, 1))
    box = tuple(torch.from_numpy(a).to(dev) for a in (low[system], high[system], there))
    # kn, en, muc, kt of every system, for pairs and walls
    values = np.array([[[law[3][0], law[3][1], law[3][3], law[3][4]] for law in laws] for laws in sc.laws])
    table = torch.from_numpy(values).to(dev)  # (systems, 2, 4)
    st = torch.from_numpy(system).to(dev)
    x, v, w = (torch.from_numpy(np.ascontiguousarray(p[k])).to(dev) for k in ("position", "velocity", "omega"))
    steps, dt, fluid = case["steps"], sc.dt, None
    reach = 0.3 * MM if kind in ("bed", "app", "fluid") else 1.7 * MM  # how far apart partners may start

    def params(rows, which):
        own = table[st[rows], which]
        return tuple(own[:, k:k + 1] for k in range(4))

    if kind == "fluid":
        weight = float(p["mass"].mean()) * 9.81
        rng = np.random.default_rng(seed + 7)
        hydro = [torch.from_numpy(a).to(dev) for a in (rng.normal(0.0, 0.3 * weight, (n, 3)),
                                                       rng.normal(0.0, 0.1 * weight * MM, (n, 3)))]
        fluid = (1000.0 / RHO, *hydro)
        dt = (steps + 0.5) * dt / steps
    if kind != "adjoint":
        with torch.no_grad():
            out = _leapfrog(sc, steps, dt, params, box, x, v, w, reach, fluid)
        return {k: a.cpu().numpy() for k, a in out.items()} | {"coordination": None}
    for a in (x, v, w, table):
        a.requires_grad_(True)
    out = _leapfrog(sc, steps, dt, params, box, x, v, w, reach)
    rng = np.random.default_rng(seed + 7)
    loss = sum((out[k] * torch.from_numpy(rng.normal(0.0, 1.0, (n, 3))).to(dev)).sum()
               for k in ("position", "velocity", "omega"))
    gx, gv, gw, gt = torch.autograd.grad(loss, (x, v, w, table))
    laws = np.zeros((16, 4))  # 4 x 4 materials: sphere-sphere in slot 0, sphere-wall in slot 1
    laws[:2] = gt[0].cpu().numpy()
    return {"final": {k: out[k].detach().cpu().numpy() for k in ("position", "velocity", "omega")},
            "gradient": {"position": gx.cpu().numpy(), "velocity": gv.cpu().numpy(), "omega": gw.cpu().numpy(),
                         "laws": laws}}
