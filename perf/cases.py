"""Performance cases: the work a program has this framework do, through its
public entry points, on synthetic plates and point sets.

Kinds of case
-------------
``simulate``  one ``Model.simulate`` call with host arrays in and out, the
              model kept between calls (parameter studies call it many times
              with other material samples and initial states).
``batch``     one run of a ``BatchedSimulation`` (reset, run, results).
``adjoint``   one forward and backward pass of the differentiable rollout.
``families``  the bond families of a point set (model set-up).

Plates are regular lattices of spacing ``DX`` (optionally jittered into
irregular points) pulled apart along x, with the bulk modulus, density and
damping of the repository's benchmark.  What differs between seeds is what
differs between the samples of a study: the material parameters, the initial
displacement and velocity fields, the noise.
"""
import functools
import math
import os
import tempfile
import warnings

import numpy as np
import torch

import probabilistic_peridynamics_gb300 as pp
from probabilistic_peridynamics_gb300 import batch, lattice
from probabilistic_peridynamics_gb300.adjoint import AdjointProblem, rollout
from probabilistic_peridynamics_gb300.mesh import write_vtk
from probabilistic_peridynamics_gb300.neighbours import neighbour_family
from probabilistic_peridynamics_gb300.pointset import (nlinear_tables,
                                                       trilinear)

DX = 0.005
BULK = 1e9
S0 = 0.005
DENSITY = 2400.0
DAMPING = 2.5e6
DT = 1e-6

#: Fields of a ``simulate`` case and what most cases have.
SIMULATE = dict(kind="simulate", nx=0, ny=0, nz=0, horizon=3.015, jitter=False,
                integrator="velocity_verlet", precision="float64", steps=0,
                damage="pmb", compensated=False, crack=False, strain=0.1,
                load="pull", write=0)


def _simulate(name, **fields):
    return dict(SIMULATE, name=name, **fields)


def listed():
    return [
        # The smallest study: the reference's example is a 2-D plate of 2113
        # nodes under an edge load.  Launches and latency count.
        _simulate("plate_2d_2k_force_f64", nx=46, ny=46, nz=1,
                  integrator="euler_cromer", steps=400, load="force"),
        # The small plain-method configuration (20 x 20 x 5, Euler).
        _simulate("block_2k_euler_f64", nx=20, ny=20, nz=5,
                  integrator="euler", steps=1000),
        # An ordinary run that watches its result: bonds break, every 50
        # steps a mesh file and the recorded sums are written.
        _simulate("plate_12k_fracture_writes_f64", nx=61, ny=50, nz=4,
                  steps=200, crack=True, strain=0.8, write=50),
        # A wide horizon (rows of 256 slots) on an odd-sized block.
        _simulate("block_17k_wide_f64", nx=33, ny=27, nz=19, horizon=4.015,
                  integrator="euler_cromer", steps=100),
        # The large plain-method plate in the default precision.
        _simulate("plate_400k_vv_f64", nx=200, ny=200, nz=10, steps=150,
                  crack=True),
        # The same plate in mixed precision: the headline configuration.
        _simulate("plate_400k_vv_mixed", nx=200, ny=200, nz=10, steps=1000,
                  precision="mixed", crack=True),
        # Fracture in mixed precision: released close to the critical strain.
        _simulate("plate_100k_fracture_mixed", nx=199, ny=101, nz=5,
                  steps=400, precision="mixed", crack=True, strain=0.8),
        # Irregular points, three bond types, trilinear damage, compensated.
        _simulate("composite_250k_mixed", nx=200, ny=125, nz=10,
                  horizon=2.1, jitter=True, steps=200, precision="mixed",
                  damage="trilinear", compensated=True, strain=0.75),
        # The same material in the default precision.
        _simulate("composite_31k_f64", nx=83, ny=53, nz=7, horizon=2.1,
                  jitter=True, steps=100, damage="trilinear", strain=0.75),
        # PeriPy's CPU integrator, whose sequential results are kept.
        _simulate("plate_29k_cpu_euler", nx=60, ny=60, nz=8,
                  integrator="cpu_euler", steps=60),
        # Uncertainty quantification: uneven plates stepped together.
        dict(name="uq_6_plates_mixed", kind="batch", count=6, nx_lo=40,
             nx_hi=160, nz=5, precision="mixed", steps=200),
        # Gradients with respect to every bond's stiffness.
        dict(name="adjoint_12k", kind="adjoint", nx=50, ny=50, nz=5,
             steps=500, every=50, dtype="float32"),
    ]


#: Rows of 32, 128 and 256 slots in three dimensions, 32, 64 and 128 in two.
_HORIZONS = {True: (3.015, 4.015, 5.015), False: (2.015, 3.015, 4.015)}


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _neighbours(horizon, flat):
    """About how many neighbours a node has."""
    return math.pi * horizon ** 2 if flat else 4.19 * horizon ** 3


def draw(rng):
    kind = rng.choice(["simulate"] * 7 + ["batch", "adjoint", "families"])
    if kind == "batch":
        lo = rng.randint(20, 60)
        return dict(kind=kind, count=rng.randint(2, 7), nx_lo=lo,
                    nx_hi=lo + rng.randint(5, 90), nz=rng.randint(2, 5),
                    precision=rng.choice(["mixed", "mixed", "float64"]),
                    steps=rng.randint(10, 40))
    if kind == "adjoint":
        return dict(kind=kind, nx=rng.randint(9, 60), ny=rng.randint(9, 50),
                    nz=rng.randint(3, 5), steps=rng.randint(20, 120),
                    every=rng.choice([10, 25, 50]),
                    dtype=rng.choice(["float32", "float64"]))
    if kind == "families":
        return dict(kind=kind, nodes=_log_uniform(rng, 1000, 300_000),
                    horizon=rng.choice(_HORIZONS[False]))
    flat = rng.random() < 0.2
    horizon = rng.choice(_HORIZONS[flat])
    integrator = rng.choice(["euler", "euler_cromer", "velocity_verlet",
                             "velocity_verlet", "cpu_euler"])
    cpu = integrator == "cpu_euler"
    precision = "float64" if cpu else rng.choice(["float64", "mixed"])
    mixed = precision == "mixed"
    nodes = _log_uniform(rng, 1000, 30_000 if cpu else 250_000)
    if flat:
        nx = max(9, int(math.sqrt(nodes) * rng.uniform(0.6, 1.6)))
        ny, nz = max(9, nodes // nx), 1
    else:
        nz = rng.randint(3, 11)
        nx = max(9, int(math.sqrt(nodes / nz) * rng.uniform(0.6, 1.6)))
        ny = max(9, nodes // (nz * nx))
    # as many steps as a bounded amount of bond work gives
    bonds = nx * ny * nz * _neighbours(horizon, flat)
    steps = int(min(500, (1.5e10 if mixed else 1.5e9) / bonds))
    steps = max(10, int(steps * rng.uniform(0.3, 1.0)))
    jitter = not flat and not cpu and rng.random() < 0.4
    if jitter:
        horizon -= 0.2
    damage = ("trilinear" if not cpu and not flat and rng.random() < 0.3
              else "pmb")
    case = dict(SIMULATE, nx=nx, ny=ny, nz=nz, horizon=horizon, jitter=jitter,
                integrator=integrator, precision=precision, steps=steps,
                damage=damage, compensated=mixed and rng.random() < 0.3,
                crack=rng.random() < 0.5,
                strain=rng.choice([0.1, 0.1, 0.5]),
                load="pull" if cpu else rng.choice(["pull", "pull", "force"]))
    return case


# ------------------------------------------------------------ the material
def _stiffness(case, bulk=BULK):
    """Micro-modulus: 3-D, or a plate one spacing thick."""
    h = case["horizon"] * DX
    if case["nz"] == 1:
        return 9.0 * bulk / (math.pi * DX * h ** 3)
    return lattice.bond_stiffness_pmb(bulk, h)


def _dt(case):
    """A stable step: the explicit Euler update of u by f needs one below
    2 / lambda_max, lambda_max <= 2 sum_j c vol / |xi|."""
    if case["integrator"] in ("euler", "cpu_euler"):
        return 0.5 * (case["horizon"] * DX) ** 2 / (72.0 * BULK)
    return DT


def _tables(case, k, s0):
    """(bond_stiffness, critical_stretch) of the damage model: one bond type
    (PMB), or two materials and their interface with trilinear softening."""
    if case["damage"] == "pmb":
        return float(k), float(s0)
    mean = 2.0 * k * 3.0 * k / (k + 3.0 * k)
    rows = [trilinear(c, 0.8 * s0, 1.2 * s0, 2.0 * s0)
            for c in (k, 3.0 * k, mean)]
    return np.array([r[0] for r in rows]), np.array([r[1] for r in rows])


# ------------------------------------------------------------ the geometry
def _points(case):
    coords = lattice.lattice_coords(case["nx"], case["ny"], case["nz"], DX)
    if case["jitter"]:
        coords = coords + DX * np.random.default_rng(7).uniform(
            -0.25, 0.25, coords.shape)
    return coords


def _crack(coords, nlist, n_neigh):
    """Bonds across the middle plane below a quarter of the height."""
    x, y = coords[:, 0], coords[:, 1]
    mid = 0.5 * (x.min() + x.max()) + 1e-4 * DX
    return lattice.plane_crack_pairs(coords, nlist, n_neigh, mid,
                                     y.min() + 0.25 * np.ptp(y))


@functools.lru_cache(maxsize=4)
def _model(key):
    """The model a program keeps between ``simulate`` calls."""
    case = dict(key)
    coords = _points(case)
    n = coords.shape[0]
    x = coords[:, 0]
    lo, hi = x.min() + 0.6 * DX, x.max() - 0.6 * DX
    pull = case["load"] == "pull"

    def displacement(p):
        if p[0] <= lo:
            return [-1.0 if pull else 0.0, None, None]
        if pull and p[0] >= hi:
            return [1.0, None, None]
        return [None, None, None]

    def force(p):
        if not pull and p[0] >= hi:
            return [1.0, None, None]
        return [None, None, None]

    def tip(p):
        return ["tip" if p[0] >= hi else None, None, None]

    kinds = dict(euler=pp.EulerCUDA, euler_cromer=pp.EulerCromerCUDA,
                 velocity_verlet=pp.VelocityVerletCUDA)
    if case["integrator"] == "cpu_euler":
        integrator = pp.Euler(_dt(case))
    else:
        args = () if case["integrator"] == "euler" else (DAMPING,)
        options = (dict(precision="mixed", compensated=case["compensated"])
                   if case["precision"] == "mixed" else {})
        integrator = kinds[case["integrator"]](*args, dt=_dt(case), **options)
    horizon = case["horizon"] * DX
    k, s = _tables(case, _stiffness(case), S0)
    more = {}
    if case["damage"] != "pmb":
        family, nlist, _ = neighbour_family(coords, horizon,
                                            integrator.context)
        left = x < 0.5 * (x.min() + x.max())
        other = left[np.where(nlist >= 0, nlist, 0)]
        types = np.where(left[:, None] & other, 0,
                         np.where(left[:, None] | other, 2, 1))
        types = np.where(nlist >= 0, types, 0).astype(np.intc)
        more = dict(family=family, connectivity=(nlist, family.copy()),
                    bond_types=types)
    elif case["crack"]:
        more = dict(initial_crack=_crack)
    with tempfile.TemporaryDirectory() as folder, warnings.catch_warnings():
        warnings.simplefilter("ignore")
        mesh = os.path.join(folder, "points.vtk")
        write_vtk(mesh, coords, [])
        return pp.Model(
            mesh, integrator, horizon=horizon, critical_stretch=s,
            bond_stiffness=k, transfinite=1, volume_total=n * DX ** 3,
            dimensions=2 if case["nz"] == 1 else 3,
            is_displacement_boundary=displacement, is_force_boundary=force,
            is_tip=tip, density=(np.full(n, DENSITY) if case["integrator"]
                                 in ("euler_cromer", "velocity_verlet")
                                 else None), **more)


def _key(case):
    """What the model depends on."""
    return tuple(sorted((f, case[f]) for f in SIMULATE
                        if f not in ("kind", "steps", "strain", "write")))


def _field(rng, coords, amplitude):
    """A smooth displacement field with some noise from node to node."""
    u = np.zeros_like(coords)
    span = np.maximum(np.ptp(coords, axis=0), DX)
    for _ in range(4):
        wave = rng.integers(1, 4, 3) * math.pi / span
        phase = rng.uniform(0, 2 * math.pi)
        direction = rng.normal(size=3)
        u += direction * np.sin(coords @ wave + phase)[:, None]
    u *= amplitude
    return u + rng.normal(scale=1e-3 * amplitude, size=u.shape)


# ---------------------------------------------------------------- prepare
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    return _PREPARE[case["kind"]](case, rng)


def _prepare_simulate(case, rng):
    model = _model(_key(case))
    coords = model.coords
    x = coords[:, 0]
    # strained along x to the given share of the critical stretch, with a
    # smooth field and noise on top; pulled plates are strained about their
    # middle and their faces start where that puts them, clamped ones about
    # the clamped face
    pull = case["load"] == "pull"
    origin = 0.5 * (x.min() + x.max()) if pull else x.min()
    strain = case["strain"] * S0
    u = _field(rng, coords, 0.02 * strain * DX)
    u[:, 0] += strain * (x - origin)
    if case["nz"] == 1:
        u[:, 2] = 0.0
    k, s = _tables(case, _stiffness(case) * rng.uniform(0.95, 1.05),
                   S0 * rng.lognormal(0.0, 0.02))
    ramp = np.arange(1, case["steps"] + 1)
    state = dict(model=model, steps=case["steps"], u=u,
                 ud=rng.normal(scale=1e-4, size=u.shape),
                 bond_stiffness=k, critical_stretch=s,
                 displacement=(strain * (x.max() - origin) + 1e-8 * ramp
                               if pull else None),
                 force=None if pull else 1e-2 * ramp,
                 write=case["write"] or None)
    if case["integrator"] in ("euler", "cpu_euler"):
        state["ud"] = None
    if case["write"]:
        state["folder"] = tempfile.TemporaryDirectory()
    return state


def _prepare_batch(case, rng):
    instances = []
    # the plates' sizes belong to the case, their material to the seed
    sizes = np.random.default_rng([case["count"], case["nx_hi"]]).integers(
        case["nx_lo"], case["nx_hi"] + 1, (case["count"], 2))
    for nx, ny in sizes:
        coords = lattice.lattice_coords(nx, ny, case["nz"], DX)
        n = coords.shape[0]
        family, nlist, _ = neighbour_family(coords, 3.015 * DX,
                                            _context())
        bc_types, bc_values = lattice.face_bcs(coords, 0)
        # stiffness noise, uniform in 0.9 .. 1.1, equal for both directions
        phase = rng.uniform(size=n)
        noise = phase[:, None] + phase[nlist]
        noise -= np.floor(noise)
        instances.append(batch.Instance(
            coords=coords, volume=np.full(n, DX ** 3), family=family,
            nlist=nlist, n_neigh=family.copy(), bc_types=bc_types,
            bc_values=bc_values, densities=np.full((n, 3), DENSITY),
            critical_stretch=float(rng.lognormal(math.log(S0), 0.2)),
            stiffness_corrections=0.9 + 0.2 * noise))
    options = dict(precision="mixed") if case["precision"] == "mixed" else {}
    simulation = batch.BatchedSimulation(
        batch.concatenate(instances),
        pp.EulerCromerCUDA(DAMPING, dt=DT, **options),
        lattice.bond_stiffness_pmb(BULK, 3.015 * DX))
    return dict(simulation=simulation, steps=case["steps"],
                displacement=2e-8 * np.arange(1, case["steps"] + 1))


@functools.lru_cache(maxsize=1)
def _context():
    return pp.CUDAContext(0)


@functools.lru_cache(maxsize=4)
def _problem(nx, ny, nz, steps):
    """The adjoint problem of a block of unit spacing."""
    coords = lattice.lattice_coords(nx, ny, nz, 1.0)
    family, nlist, _ = lattice.lattice_family(nx, ny, nz, 3.015)
    bc_types, bc_values = lattice.face_bcs(coords, 0)
    return nlist, AdjointProblem(coords, np.ones(len(coords)), nlist, bc_types,
                                 bc_values, 1e-6 * np.arange(1, steps + 1),
                                 0.5)


def _prepare_adjoint(case, rng):
    nlist, problem = _problem(case["nx"], case["ny"], case["nz"],
                              case["steps"])
    n = nlist.shape[0]
    phase = rng.uniform(size=n)
    noise = phase[:, None] + phase[nlist]
    k = np.where(nlist >= 0, 0.01 * (0.9 + 0.2 * (noise - np.floor(noise))),
                 0.0)
    return dict(problem=problem, steps=case["steps"], every=case["every"],
                k=torch.tensor(k, dtype=getattr(torch, case["dtype"]),
                               device="cuda", requires_grad=True),
                probes=torch.tensor(rng.choice(n, min(100, n // 4),
                                               replace=False), device="cuda"))


def _prepare_families(case, rng):
    # uniform points at the lattice's density
    edge = DX * case["nodes"] ** (1.0 / 3.0)
    return dict(coords=rng.uniform(0.0, edge, (case["nodes"], 3)),
                horizon=case["horizon"] * DX, context=_context())


_PREPARE = dict(simulate=_prepare_simulate, batch=_prepare_batch,
                adjoint=_prepare_adjoint, families=_prepare_families)


# -------------------------------------------------------------------- run
def run(state):
    if "model" in state:
        return _run_simulate(state)
    if "simulation" in state:
        return _run_batch(state)
    if "problem" in state:
        return _run_adjoint(state)
    family, nlist, _ = neighbour_family(state["coords"], state["horizon"],
                                        state["context"])
    return dict(family=family, nlist=nlist)


def _run_simulate(state):
    ud = state["ud"]
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")  # "over 5% of bonds have broken"
        u, damage, (nlist, n_neigh), force, ud, data = \
            state["model"].simulate(
                state["steps"], u=state["u"].copy(),
                ud=None if ud is None else ud.copy(),
                bond_stiffness=state["bond_stiffness"],
                critical_stretch=state["critical_stretch"],
                displacement_bc_magnitudes=state["displacement"],
                force_bc_magnitudes=state["force"], write=state["write"],
                write_path=(state["folder"].name if state["write"]
                            else None))
    return dict(u=u, ud=ud, force=force, damage=damage, nlist=nlist,
                n_neigh=n_neigh, data=data)


def _run_batch(state):
    simulation = state["simulation"]
    simulation.reset()
    simulation.run(state["steps"], state["displacement"])
    return [dict(u=u, ud=ud, damage=damage, nlist=nlist, n_neigh=n_neigh)
            for u, ud, damage, nlist, n_neigh in simulation.results()]


def _run_adjoint(state):
    k = state["k"]
    k.grad = None
    u = rollout(k, 1.0, state["problem"], state["steps"], state["every"])
    loss = (u[state["probes"]] ** 2).sum()
    loss.backward()
    return dict(u=u.detach(), loss=loss.detach(), grad=k.grad)


# ------------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass.  A step reads each bond's neighbour
    index (and type, regime and correction where there are some) and each
    node's arrays once, in the layouts of the reference's kernels, and writes
    the node's new state; about 40 operations a bond."""
    kind = case["kind"]
    if kind == "families":
        n = case["nodes"]
        bonds = n * _neighbours(case["horizon"], False)
        return dict(bytes=24 * n + 4 * n + 4 * bonds, flops=8 * 6.4 * bonds)
    if kind == "batch":
        mean = 0.5 * (case["nx_lo"] + case["nx_hi"])
        n = case["count"] * mean * mean * case["nz"]
        return dict(bytes=case["steps"] * n * (336 + 100 * 12),
                    flops=case["steps"] * n * 100 * 40)
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "adjoint":
        # forward, recomputed forward and reverse steps
        bonds = n * 90
        return dict(bytes=case["steps"] * (2 * (bonds * 12 + n * 216)
                                           + bonds * 28 + n * 100),
                    flops=case["steps"] * bonds * (2 * 40 + 70))
    bonds = n * _neighbours(case["horizon"], case["nz"] == 1)
    node = 336 if case["integrator"] in ("euler_cromer",
                                         "velocity_verlet") else 216
    bond = 4 if case["damage"] == "pmb" else 12
    return dict(bytes=case["steps"] * (bonds * bond + n * node),
                flops=case["steps"] * bonds * 40)


# ------------------------------------------------------------------ exact
#: Bond slots times steps that the 64-bit restatement takes on.
_EXACT_MOST = 2.0e10


def exact(case, seed):
    kind = case["kind"]
    if kind == "families":
        return None  # whole numbers
    state = prepare(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, state)
    if kind == "batch":
        return _exact_batch(state)
    return _exact_simulate(case, state)


def _f64(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")


class _Rows:
    """Bonds of a model as (nodes, slots) tensors, in 64 bits."""

    def __init__(self, coords, volume, nlist, n_neigh, corrections=None):
        self.r0 = _f64(coords)
        self.volume = _f64(volume)
        nlist = torch.as_tensor(np.asarray(nlist), device="cuda").long()
        slot = torch.arange(nlist.shape[1], device="cuda")
        count = torch.as_tensor(np.asarray(n_neigh), device="cuda")
        self.live = (nlist >= 0) & (slot < count[:, None])
        self.j = torch.where(self.live, nlist, 0)
        self.corrections = None if corrections is None else _f64(corrections)

    def force(self, u, law):
        """Force of every node; ``law(a, b, stretch)`` gives the bond force
        over the rows a .. b and drops the bonds that break from ``live``."""
        out = torch.empty_like(u)
        n, width = self.j.shape
        size = max(1, 20_000_000 // width)
        for a in range(0, n, size):
            b = min(n, a + size)
            j = self.j[a:b]
            xi = self.r0[j] - self.r0[a:b, None]
            p = xi + (u[j] - u[a:b, None])
            length = xi.square().sum(-1).sqrt()
            y = p.square().sum(-1).sqrt()
            f = law(a, b, (y - length) / length)
            if self.corrections is not None:
                f = f * self.corrections[a:b]
            f = torch.where(self.live[a:b], f * self.volume[j] / y, 0.0)
            out[a:b] = (f[..., None] * torch.where(self.live[a:b, :, None], p,
                                                   0.0)).sum(1)
        return out


def _march(rows, law, integrator, dt, steps, u, ud, bc, disp, fbc, fmag):
    """``steps`` steps; returns u, ud and the last force."""
    types, values = (torch.as_tensor(np.asarray(a), device="cuda")
                     for a in bc)
    held = types != 0
    udd = torch.zeros_like(u)
    f = None
    for t in range(steps):
        f = rows.force(u, law)
        if fbc is not None:
            f = torch.where(fbc[0] != 0, f + fmag[t] * fbc[1], f)
        if integrator in ("euler", "cpu_euler"):
            new = u + dt * f
        elif integrator == "euler_cromer":
            udd = (f - DAMPING * ud) / DENSITY
            ud = ud + dt * udd
            new = u + dt * ud
        else:
            half = ud + 0.5 * dt * udd
            udd = (f - DAMPING * half) / DENSITY
            ud = half + 0.5 * dt * udd
            new = u + dt * (ud + 0.5 * dt * udd)
        u = torch.where(held, disp[t] * values, new)
    return u, ud, f


def _host(t):
    return t.cpu().numpy()


def _exact_simulate(case, state):
    model = state["model"]
    nlist, n_neigh = model.initial_connectivity
    if nlist.size * case["steps"] > _EXACT_MOST:
        return None
    rows = _Rows(model.coords, model.volume, nlist, n_neigh)
    two_sided = case["integrator"] == "cpu_euler"
    k, s = state["bond_stiffness"], state["critical_stretch"]
    if case["damage"] == "pmb":
        def law(a, b, stretch):
            rows.live[a:b] &= (stretch.abs() if two_sided else stretch) < s
            return k * stretch
    else:
        k, s, c = (_f64(t) for t in nlinear_tables(k, s))
        types = torch.as_tensor(model.bond_types, device="cuda").long()
        regime = torch.zeros_like(types)

        def law(a, b, stretch):
            ty, r = types[a:b], regime[a:b]
            last = s.shape[1] - 1
            below = stretch < s[ty, r.clamp(max=last)]
            back = below & (r > 0) & (stretch < s[ty, (r - 1).clamp(min=0)])
            r = torch.where(below, torch.where(back, r - 1, r), r + 1)
            r = torch.where(rows.live[a:b], r, regime[a:b])
            regime[a:b] = r
            rows.live[a:b] &= r <= last
            r = r.clamp(max=last)
            return k[ty, r] * stretch + c[ty, r]
    steps = case["steps"]
    zero = np.zeros(steps)
    disp = state["displacement"] if state["displacement"] is not None else zero
    fmag = state["force"] if state["force"] is not None else zero
    fbc = [torch.as_tensor(np.asarray(a), device="cuda")
           for a in (model.force_bc_types, model.force_bc_values)]
    u0 = _f64(state["u"])
    ud0 = (torch.zeros_like(u0) if state["ud"] is None else _f64(state["ud"]))
    u, ud, f = _march(rows, law, case["integrator"], _dt(case), steps, u0,
                      ud0, (model.bc_types, model.bc_values), disp, fbc, fmag)
    family = _f64(model.family)
    damage = 1.0 - rows.live.sum(1) / family
    return dict(u=_host(u), ud=_host(ud), force=_host(f),
                damage=_host(damage), nlist=None, n_neigh=None, data=None)


def _exact_batch(state):
    b = state["simulation"].batch
    if b.nlist.size * state["steps"] > _EXACT_MOST:
        return None
    rows = _Rows(b.coords, b.volume, b.nlist, b.n_neigh,
                 b.stiffness_corrections)
    s = _f64(b.instance_s0)[torch.as_tensor(b.node_instance,
                                            device="cuda").long()]
    k = state["simulation"].bond_stiffness

    def law(lo, hi, stretch):
        rows.live[lo:hi] &= stretch < s[lo:hi, None]
        return k * stretch

    zero = torch.zeros_like(rows.r0)
    u, ud, _ = _march(rows, law, "euler_cromer", DT, state["steps"], zero,
                      zero, (b.bc_types, b.bc_values), state["displacement"],
                      None, None)
    damage = 1.0 - rows.live.sum(1) / _f64(b.family)
    u, ud, damage = (_host(a) for a in (u, ud, damage))
    return [dict(u=x, ud=v, damage=d, nlist=None, n_neigh=None)
            for x, v, d in zip(b.split(u), b.split(ud), b.split(damage))]


def _exact_adjoint(case, state):
    """The rollout and its gradient by autograd, in 64 bits."""
    from torch.utils.checkpoint import checkpoint
    problem = state["problem"]
    nlist, _ = _problem(case["nx"], case["ny"], case["nz"], case["steps"])
    coords = lattice.lattice_coords(case["nx"], case["ny"], case["nz"], 1.0)
    bc_types, bc_values = lattice.face_bcs(coords, 0)
    r0 = _f64(coords)
    live = torch.as_tensor(nlist >= 0, device="cuda")
    j = torch.as_tensor(np.where(nlist >= 0, nlist, 0), device="cuda").long()
    # a slot without a bond points one unit away, so that no gradient is NaN
    xi = torch.where(live[..., None], r0[j] - r0[:, None],
                     torch.ones(3, dtype=torch.float64, device="cuda"))
    length = xi.square().sum(-1).sqrt()
    held = torch.as_tensor(bc_types != 0, device="cuda")
    values = _f64(bc_values)
    k = state["k"].detach().double().requires_grad_(True)

    def segment(u, k, t0, t1):
        for t in range(t0, t1):
            du = torch.where(live[..., None], u[j] - u[:, None], 0.0)
            p = xi + du
            y = p.square().sum(-1).sqrt()
            f = torch.where(live, k * (y - length) / length / y, 0.0)
            new = u + problem.dt * (f[..., None] * p).sum(1)
            u = torch.where(held, float(problem.mags[t]) * values, new)
        return u

    u = torch.zeros_like(r0)
    for t0 in range(0, case["steps"], 25):
        u = checkpoint(segment, u, k, t0, min(t0 + 25, case["steps"]),
                       use_reentrant=False)
    loss = (u[state["probes"]] ** 2).sum()
    loss.backward()
    return dict(u=_host(u.detach()), loss=float(loss), grad=_host(k.grad))
