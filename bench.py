#!/usr/bin/env python
"""Headline benchmark: bond-updates/s of the fused mixed-precision step.

Workload (the large plain-method configuration): a 200 x 200 x 10 regular
lattice, dx = 0.005 (a 1 x 1 x 0.05 plate), horizon 3.015 dx, node volume
dx^3, PMB bonds with c = 18 K / (pi delta^4), K = 1e9, s0 = 0.005; a
pre-crack removes every bond crossing the plane x = 0.5 at y < 0.25; the
x-min and x-max faces are pulled apart by 1e-8 per step; Velocity-Verlet
with density 2400, damping 2.5e6 and dt = 1e-6.  400,000 nodes and
42,700,528 directed bonds (one bond-update = one directed family bond in
one step, counted on the initial connectivity).

Arms
----
``python bench.py [--gpus N] [--steps K] [--warmup W]``
    Our CUDA step.  ``value`` is the device-timed fused mixed-precision
    (FP32 bonds, exact FP64 stretch test, double-float state) throughput
    with the state resident in HBM; the plain and fused FP64 steps are timed
    beside it (``variants``), the displacement error of the mixed step
    against the FP64 step and the broken-bond mask are stated
    (``accuracy``), ``e2e`` is a full 5000-step ``Model.simulate`` through
    the public API with host arrays in and out, ``roofline`` relates the
    fused kernel to the measured HBM bandwidth and ``cpu_baseline`` is the
    reference's own CPU step timed on the host.
``python bench.py --impl reference ...``
    The reference's own CPU step (``peripy/peridynamics.pyx`` break_bonds +
    bond_force + update_displacement, as ``Euler.__call__`` calls them),
    compiled from its sources into ``oracle/_ref``, on a bounded block
    (4 x ny x 10) of the same lattice per step, pulled at the plate's strain
    rate, with a stable Euler pseudo-step (see ``CPU_DT``).

Under torchrun every rank runs an independent replica on its own GPU (the
configuration fits one GPU); ``value`` is the sum over ranks.
"""
import argparse
import json
import os
import pathlib
import statistics
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = pathlib.Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = ("bond-updates/sec at 1 GB300, FP32 fused vs FP64 plain at stated "
          "disp. error")
UNIT = "bond-updates/s"
WORKLOAD = ("pre-cracked 200x200x10 lattice, 400k nodes, 42.7M bonds, "
            "Velocity-Verlet")
NX, NY, NZ = 200, 200, 10
DX = 0.005
HORIZON_CELLS = 3.015
BULK_MODULUS = 1e9
S0 = 0.005
DENSITY = 2400.0
DAMPING = 2.5e6
DT = 1e-6
PULL_RATE = 1e-8
E2E_STEPS = 5000
#: reference-layout bytes per directed bond (int32 nlist read) and per node
#: for Velocity-Verlet: reads u 24, r0 24, vol 8, bc_types 12, bc_values 24,
#: force_bc_types 12, force_bc_values 24, family 4, ud 24, udd 24,
#: densities 24; writes u 24, force 24, body_force 24, damage 8, n_neigh 4,
#: ud 24, udd 24.
B_BOND = 4
B_NODE_VV = 336


def parse_args():
    p = argparse.ArgumentParser(description=__doc__.split("\n")[0])
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=20000)
    p.add_argument("--warmup", type=int, default=20)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--fp64-steps", type=int, default=10,
                   help="timed steps of each FP64 variant")
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu", action="store_true")
    p.add_argument("--no-variants", action="store_true",
                   help="skip the batched, composite and adjoint timings")
    p.add_argument("--accuracy-steps", type=int, default=E2E_STEPS)
    p.add_argument("--workload",
                   choices=["large", "batched", "composite", "adjoint",
                            "writes", "setup"],
                   default="large",
                   help="large: the 200x200x10 Velocity-Verlet plate (the "
                        "headline); batched: 64 uneven UQ instances, "
                        "Euler-Cromer; composite: 1M Poisson-disk points, "
                        "three bond types, trilinear damage; adjoint: "
                        "forward + backward passes of the 50x50x5 rollout; "
                        "writes: Model.simulate of the plate with a write "
                        "every 500 steps, device sums against host copies; "
                        "setup: neighbour families and initial crack of the "
                        "plate, GPU against host and the reference")
    p.add_argument("--profile", choices=["mixed", "fp64", "plain",
                                         "composite", "batched"],
                   help="only run 3 warm-up and 3 profiled launches of one "
                        "step variant on the full workload (for ncu)")
    return p.parse_args()


def profile_case(which):
    """3 warm-up + 3 launches of one step variant, direct launches."""
    import torch
    if which == "composite":
        profile_composite()
        return
    if which == "batched":
        profile_batched()
        return
    w = build_workload()
    precision = "mixed" if which == "mixed" else "float64"
    if which == "mixed":
        # PP_PROFILE_TILED=0: the untiled kernel (k_mixed), else k_tiled
        tiled = os.environ.get("PP_PROFILE_TILED", "1") != "0"
        import probabilistic_peridynamics_gb300 as pp
        integ = pp.VelocityVerletCUDA(DAMPING, dt=DT, precision="mixed",
                                      autotune=False, tiled=tiled)
        integ.build(w["nnodes"], 3, w["max_neigh"], w["coords"],
                    w["volume"], w["family"], w["bc_types"], w["bc_values"],
                    w["force_bc_types"], w["force_bc_values"], None, None,
                    w["densities"])
        z = np.zeros((w["nnodes"], 3))
        integ.create_buffers(w["nlist"], w["n_neigh"], w["k"], w["s0"], None,
                             z, z, z, z, z, np.zeros(w["nnodes"]), None, 1, 1)
        integ._fargs.variant = int(os.environ.get(
            "PP_PROFILE_VARIANT", "1"))
    else:
        integ = make_integrator(w, precision, which != "plain",
                                autotune=False)
    for k in range(6):
        integ(PULL_RATE * (k + 1), 0.0)
    integ.context.stream.synchronize()
    torch.cuda.synchronize()
    print(f"profile case {which}: 6 steps done", flush=True)


def profile_composite():
    """3 warm-up + 3 launches of the composite's mixed step (compensated
    sums, the tile shape of PP_PROFILE_VARIANT, default 2)."""
    import torch
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300.integrators import CUDAContext
    from probabilistic_peridynamics_gb300.pointset import composite
    w = composite(context=CUDAContext(0))
    n = w["coords"].shape[0]
    tiled = os.environ.get("PP_PROFILE_TILED", "1") != "0"
    integ = pp.VelocityVerletCUDA(DAMPING, dt=DT, precision="mixed",
                                  compensated=True, autotune=False,
                                  tiled=tiled)
    integ.build(n, 3, w["max_neigh"], w["coords"], w["volume"], w["family"],
                w["bc_types"], w["bc_values"], np.zeros((n, 3), dtype=np.intc),
                np.zeros((n, 3)), None, w["bond_types"], w["densities"])
    z = np.zeros((n, 3))
    integ.create_buffers(w["nlist"], w["n_neigh"], w["bond_stiffness"],
                         w["critical_stretch"], w["plus_cs"], z, z, z, z, z,
                         np.zeros(n), None, w["nregimes"], w["nbond_types"])
    integ._fargs.variant = int(os.environ.get("PP_PROFILE_VARIANT", "2"))
    for k in range(6):
        integ(COMPOSITE_RATE * (k + 1), 0.0)
    integ.context.stream.synchronize()
    torch.cuda.synchronize()
    print("profile case composite: 6 steps done", flush=True)


def profile_batched():
    """3 warm-up + 3 launches of the batched UQ step on 16 of the 64
    instances (the same generator: nx, ny uniform in 60..200, nz 5; about
    1.4M nodes, a few GB on the device), tiled layout, tile shape
    PP_PROFILE_VARIANT (default 1, the one the autotuner picks for the 64
    instances); no tuning launches."""
    import torch
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import batch, lattice
    b = batch.concatenate(batch.uq_instances(count=16, seed=2024, dx=DX))
    k = lattice.bond_stiffness_pmb(BULK_MODULUS, HORIZON_CELLS * DX)
    integ = pp.EulerCromerCUDA(DAMPING, dt=DT, precision="mixed",
                               autotune=False)
    sim = batch.BatchedSimulation(b, integ, k)
    integ._fargs.variant = int(os.environ.get("PP_PROFILE_VARIANT", "1"))
    for s in range(6):
        integ(PULL_RATE * (s + 1), 0.0)
    integ.context.stream.synchronize()
    torch.cuda.synchronize()
    kernel = "k_tiled" if integ.tiling is not None else "k_mixed"
    print(f"profile case batched: 6 steps done ({b.nnodes} nodes, {b.bonds}"
          f" bonds, {kernel}, variant {integ._fargs.variant})", flush=True)
    del sim


# ----------------------------------------------------------------- workload
def build_workload(pow2=True):
    from probabilistic_peridynamics_gb300 import lattice
    coords = lattice.lattice_coords(NX, NY, NZ, DX)
    family, nlist, width = lattice.lattice_family(NX, NY, NZ, HORIZON_CELLS,
                                                  pow2=pow2)
    n_neigh = family.copy()
    pairs = lattice.plane_crack_pairs(coords, nlist, n_neigh, 0.5, 0.25)
    lattice.remove_pairs(pairs, nlist, n_neigh)
    bc_types, bc_values = lattice.face_bcs(coords, 0)
    n = coords.shape[0]
    horizon = HORIZON_CELLS * DX
    return dict(coords=coords, volume=np.full(n, DX ** 3), family=family,
                nlist=nlist, n_neigh=n_neigh, bc_types=bc_types,
                bc_values=bc_values,
                force_bc_types=np.zeros((n, 3), dtype=np.intc),
                force_bc_values=np.zeros((n, 3)),
                densities=np.full((n, 3), DENSITY), nnodes=n,
                max_neigh=int(width), horizon=horizon,
                k=lattice.bond_stiffness_pmb(BULK_MODULUS, horizon), s0=S0,
                bonds=int(family.sum()), crack_pairs=int(len(pairs)))


def make_integrator(w, precision, fused, context=None, autotune=True,
                    u0=None):
    """A Velocity-Verlet integrator on the plate, from rest at ``u0``
    (default: undeformed)."""
    import probabilistic_peridynamics_gb300 as pp
    integ = pp.VelocityVerletCUDA(DAMPING, dt=DT, precision=precision,
                                  fused=fused, context=context,
                                  autotune=autotune)
    integ.build(w["nnodes"], 3, w["max_neigh"], w["coords"], w["volume"],
                w["family"], w["bc_types"], w["bc_values"],
                w["force_bc_types"], w["force_bc_values"], None, None,
                w["densities"])
    n = w["nnodes"]
    z = np.zeros((n, 3))
    integ.create_buffers(w["nlist"], w["n_neigh"], w["k"], w["s0"], None,
                         z if u0 is None else u0, z, z, z, z, np.zeros(n),
                         None, 1, 1)
    return integ


#: Fracture variant of the plate: released at rest from a uniform strain
#: FRACTURE_EPS0 along x (u_x = eps0 (x - 0.5)), the faces held at that
#: strain and pulled on at PULL_RATE per step.  The bonds cut by the
#: pre-crack leave the crack faces unbalanced; the release waves and the
#: free surfaces overload bonds near the crack tip and along the faces:
#: about 270,000 bonds break within 100 steps and 380,000 within 300.
FRACTURE_EPS0 = 0.004


def fracture_state(w, eps0=FRACTURE_EPS0):
    """``(u0, mags(steps))`` of the fracture variant."""
    x = w["coords"][:, 0]
    u0 = np.zeros((w["nnodes"], 3))
    u0[:, 0] = eps0 * (x - 0.5)
    face = eps0 * (x.max() - 0.5)

    def mags(steps):
        return face + PULL_RATE * np.arange(1, steps + 1)
    return u0, mags


# -------------------------------------------------------------------- clocks
class ClockSampler:
    """SM clock, power and throttle reasons sampled every 200 ms while the
    timed region runs.

    Each sample is one ``nvidia-smi --query-gpu`` call that exits after
    printing (a looping ``nvidia-smi -lms`` writing into a pipe buffers its
    output, and stopping it loses the buffer).  Where ``nvidia-smi`` cannot
    run, the same quantities are read through NVML (``libnvidia-ml.so.1``,
    read-only queries).  ``errors`` records why a source gave nothing.
    """

    FIELDS = ("clocks.sm,clocks.max.sm,power.draw,"
              "clocks_event_reasons.hw_slowdown,"
              "clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,"
              "clocks_event_reasons.sw_power_cap")
    NAMES = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown",
             "sw_power_cap")
    #: NVML clock-event reason bits of NAMES (nvml.h)
    NVML_BITS = (0x8, 0x40, 0x20, 0x4)

    def __init__(self, gpu_index, period_s=0.2):
        self.gpu = gpu_index
        self.period = period_s
        self.samples = []  # (sm_mhz, max_mhz, power_w, reasons)
        self.errors = []
        self._stop = threading.Event()
        self._thread = None
        self._nvml = None

    def _smi(self):
        r = subprocess.run(
            ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}",
             "--format=csv,noheader,nounits"],
            capture_output=True, text=True, timeout=5)
        if r.returncode != 0:
            raise RuntimeError(f"nvidia-smi rc {r.returncode}: "
                               f"{r.stderr.strip()[:120]}")
        parts = [x.strip() for x in r.stdout.strip().split(",")]
        reasons = {n for n, f in zip(self.NAMES, parts[3:7])
                   if f.lower().startswith("active")}
        return float(parts[0]), float(parts[1]), float(parts[2]), reasons

    def _nvml_sample(self):
        import ctypes
        if self._nvml is None:
            lib = ctypes.CDLL("libnvidia-ml.so.1")
            if lib.nvmlInit_v2() != 0:
                raise RuntimeError("nvmlInit failed")
            h = ctypes.c_void_p()
            if lib.nvmlDeviceGetHandleByIndex_v2(self.gpu,
                                                 ctypes.byref(h)) != 0:
                raise RuntimeError("nvmlDeviceGetHandleByIndex failed")
            self._nvml = (lib, h)
        lib, h = self._nvml
        sm, mx, mw = ctypes.c_uint(), ctypes.c_uint(), ctypes.c_uint()
        rs = ctypes.c_ulonglong()
        lib.nvmlDeviceGetClockInfo(h, 1, ctypes.byref(sm))      # SM clock
        lib.nvmlDeviceGetMaxClockInfo(h, 1, ctypes.byref(mx))
        lib.nvmlDeviceGetPowerUsage(h, ctypes.byref(mw))
        lib.nvmlDeviceGetCurrentClocksThrottleReasons(h, ctypes.byref(rs))
        reasons = {n for n, b in zip(self.NAMES, self.NVML_BITS)
                   if rs.value & b}
        return float(sm.value), float(mx.value), mw.value / 1e3, reasons

    def _loop(self):
        sources = [self._smi, self._nvml_sample]
        while not self._stop.is_set():
            t = time.perf_counter()
            while sources:
                try:
                    self.samples.append(sources[0]())
                    break
                except Exception as e:  # noqa: BLE001 - next source
                    self.errors.append(f"{sources[0].__name__}: {e}"[:160])
                    sources.pop(0)
            if not sources:
                return
            self._stop.wait(max(0.0, self.period - (time.perf_counter() - t)))

    def start(self):
        self._thread = threading.Thread(target=self._loop, daemon=True)
        self._thread.start()

    def stop(self):
        self._stop.set()
        if self._thread is not None:
            self._thread.join(timeout=10)
        sm = [s[0] for s in self.samples]
        loaded = [s[0] for s in self.samples if s[2] > 300.0] or sm
        reasons = set()
        for s in self.samples:
            reasons |= s[3]
        return {"sm_mhz": statistics.median(loaded) if loaded else None,
                "sm_max_mhz": max(s[1] for s in self.samples)
                if self.samples else None,
                "reasons": sorted(reasons), "samples": len(self.samples),
                "samples_under_load": sum(s[2] > 300.0 for s in self.samples),
                "power_w_max": max(s[2] for s in self.samples)
                if self.samples else None,
                "errors": self.errors[:3]}


# ------------------------------------------------------------ measurements
def job_time_ms(ms, dist, torch, device):
    """The job's time: the largest timed region over the ranks."""
    if dist is None:
        return ms
    t = torch.tensor([ms], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_throughput(world, bonds, steps, ms):
    """Bond-updates/s of the whole job: every rank steps its own replica
    of ``bonds`` bonds ``steps`` times within ``ms`` milliseconds."""
    return world * bonds * steps / (ms * 1e-3)


def time_steps(integ, steps, warmup, torch, dist=None, rate=PULL_RATE,
               offset=0.0):
    """Device time of exactly ``steps`` fused steps (graph replays); the
    displacement magnitudes are ``offset + rate * k``."""
    dm = torch.as_tensor(offset + rate * np.arange(1, warmup + steps + 1),
                         dtype=torch.float64, device=integ.context.device)
    fm = torch.zeros_like(dm)
    stream = integ.context.stream
    if warmup:
        integ._run_device(dm, fm, 0, warmup)
    stream.synchronize()
    if dist is not None:
        dist.barrier()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    integ._run_device(dm, fm, warmup, steps)
    e1.record(stream)
    e1.synchronize()
    torch.cuda.synchronize()
    if dist is not None:
        dist.barrier()
    return e0.elapsed_time(e1)


def time_kernel_launches(integ, nlaunch, torch, first_mag=0.0,
                         rate=PULL_RATE):
    """Mean duration of individual fused-step launches (events per launch)."""
    stream = integ.context.stream
    evs = [(torch.cuda.Event(enable_timing=True),
            torch.cuda.Event(enable_timing=True)) for _ in range(nlaunch)]
    for k, (a, b) in enumerate(evs):
        a.record(stream)
        integ(first_mag + rate * k, 0.0)
        b.record(stream)
    stream.synchronize()
    return statistics.mean(a.elapsed_time(b) for a, b in evs)


def time_plain_steps(integ, steps, warmup, torch):
    stream = integ.context.stream
    for k in range(warmup):
        integ(PULL_RATE * (k + 1), 0.0)
    stream.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for k in range(steps):
        integ(PULL_RATE * (warmup + k + 1), 0.0)
    e1.record(stream)
    e1.synchronize()
    return e0.elapsed_time(e1) / steps


def time_cython_euler(w, steps, torch):
    """PeriPy's CPU integrator ``Euler`` on the GPU (``pp.Euler``: the
    Cython step's semantics and results) on the bench lattice in its compact
    layout, with the CPU samples' Euler dt: the like-for-like counterpart of
    the reference CPU step that ``cpu_baseline`` times."""
    import probabilistic_peridynamics_gb300 as pp
    n = w["nnodes"]
    nl = compact(w["nlist"], w["family"])
    it = pp.Euler(CPU_DT)
    it.build(n, 3, nl.shape[1], w["coords"], w["volume"], w["family"],
             w["bc_types"], w["bc_values"], w["force_bc_types"],
             w["force_bc_values"], None, None, None)
    z = np.zeros((n, 3))
    it.create_buffers(nl, w["n_neigh"].copy(), w["k"], S0, None, z.copy(),
                      z.copy(), z.copy(), z.copy(), z.copy(), np.zeros(n),
                      None, 1, 1)
    stream = it.device_context.stream
    for k in range(2):
        it(PULL_RATE * (k + 1), 0.0)
    stream.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for k in range(steps):
        it(PULL_RATE * (k + 3), 0.0)
    e1.record(stream)
    e1.synchronize()
    ms = e0.elapsed_time(e1) / steps
    del it
    torch.cuda.empty_cache()
    return {"bond_updates_per_s": w["bonds"] / (ms * 1e-3),
            "ms_per_step": ms, "dt": CPU_DT,
            "layout": "compact rows (width family.max())"}


def accuracy(w, steps, torch):
    """Mixed vs FP64 fused (bit-identical to the plain FP64 step) after
    ``steps`` steps from the same state: displacement error and mask."""
    out = {}
    for precision in ("float64", "mixed"):
        integ = make_integrator(w, precision, True)
        mags = PULL_RATE * np.arange(1, steps + 1)
        integ._run(mags, np.zeros(steps), 0, steps)
        n = w["nnodes"]
        u, ud, udd, f, bf = (np.zeros((n, 3)) for _ in range(5))
        res = integ.write(u, ud, udd, f, bf, np.zeros(n), w["nlist"].copy(),
                          w["n_neigh"].copy())
        out[precision] = res
        del integ
        torch.cuda.empty_cache()
    u64, u32 = out["float64"][0], out["mixed"][0]
    err = float(np.max(np.abs(u32 - u64)) / np.max(np.abs(u64)))
    flips = int(np.sum(out["float64"][6] != out["mixed"][6]))
    broken = int(np.sum(w["nlist"] != -1) - np.sum(out["float64"][6] != -1))
    return {"steps": steps, "disp_rel_err_vs_fp64": err,
            "mask_flips_vs_fp64": flips, "bonds_broken_fp64": broken,
            "max_abs_u": float(np.max(np.abs(u64)))}


def _write_all(integ, w):
    n = w["nnodes"]
    z = [np.zeros((n, 3)) for _ in range(5)]
    return integ.write(*z, np.zeros(n), w["nlist"].copy(),
                       w["n_neigh"].copy())


def accuracy_fracture(w, torch, checkpoints=(100, 300)):
    """The fracture variant: mixed vs FP64 fused from the same pre-strained
    state, compared at each checkpoint step (bonds broken, mask flips,
    intact counts, displacement error)."""
    u0, mags = fracture_state(w)
    steps = max(checkpoints)
    m = mags(steps)
    out = {}
    for precision in ("float64", "mixed"):
        integ = make_integrator(w, precision, True, u0=u0)
        done, snaps = 0, {}
        for c in checkpoints:
            integ._run(m, np.zeros(steps), done, c - done)
            done = c
            snaps[c] = _write_all(integ, w)
        out[precision] = snaps
        del integ
        torch.cuda.empty_cache()
    res = {"eps0": FRACTURE_EPS0, "pull_rate": PULL_RATE}
    initial = int(np.sum(w["nlist"] != -1))
    for c in checkpoints:
        a, b = out["float64"][c], out["mixed"][c]
        res[f"step_{c}"] = {
            "bonds_broken_fp64": initial - int(np.sum(a[6] != -1)),
            "mask_flips_vs_fp64": int(np.sum(a[6] != b[6])),
            "n_neigh_equal": bool(np.array_equal(a[7], b[7])),
            "disp_rel_err_vs_fp64": float(np.max(np.abs(b[0] - a[0])) /
                                          np.max(np.abs(a[0]))),
            "max_abs_u": float(np.max(np.abs(a[0])))}
    return res


def time_fracture(w, steps, torch, ctx=None, settle=100):
    """The mixed step in the fractured state: ``settle`` steps from the
    pre-strained state (most of the breaking happens there), then
    ``steps`` graph-replayed steps timed while bonds keep breaking."""
    u0, mags = fracture_state(w)
    integ = make_integrator(w, "mixed", True, context=ctx, u0=u0)
    m = mags(settle)
    integ._run(m, np.zeros(settle), 0, settle)
    before = _write_all(integ, w)
    ms = time_steps(integ, steps, 0, torch, offset=float(m[-1]))
    kernel_ms = time_kernel_launches(integ, 50, torch,
                                     first_mag=float(m[-1]) +
                                     PULL_RATE * (steps + 1))
    after = _write_all(integ, w)
    del integ
    torch.cuda.empty_cache()
    initial = int(np.sum(w["nlist"] != -1))
    return {"bond_updates_per_s": w["bonds"] * steps / (ms * 1e-3),
            "ms_per_step": ms / steps, "kernel_ms": kernel_ms,
            "timed_steps": steps, "after_steps": settle,
            "bonds_broken_before": initial - int(np.sum(before[6] != -1)),
            "bonds_broken_after": initial - int(np.sum(after[6] != -1)),
            "eps0": FRACTURE_EPS0}


def _kernel_name(integ):
    return "k_tiled" if getattr(integ, "tiling", None) is not None \
        else "k_mixed"


def _roofline_frac(alg_bytes, kernel_ms, peak):
    return alg_bytes / (kernel_ms * 1e-3) / 1e9 / peak


def _tuning_summary(tuning):
    """The autotuner's choice against the untuned default (the tiled
    layout's tile shape 0), from its per-candidate timings."""
    if not tuning:
        return None
    best = min(tuning, key=tuning.get)
    default = "tiled/0" if "tiled/0" in tuning else "untiled/0"
    return {"chosen": best, "chosen_ms": tuning[best], "default": default,
            "default_ms": tuning[default],
            "speedup": tuning[default] / tuning[best]}


def variant_batched(torch, peak, steps=20, warmup=3):
    """The batched UQ form, briefly: 64 uneven instances (nx, ny uniform in
    60..200, nz 5), Euler-Cromer, lognormal s0, U(0.9, 1.1) bond noise,
    one persistent launch per step (graph replays), autotuned layout and
    tile shape.  Algorithmic bytes: 4 B neighbour index + 8 B binary64
    stiffness correction per bond, 336 B per node."""
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import batch, lattice
    t0 = time.perf_counter()
    inst = batch.uq_instances(count=64, seed=2024, dx=DX)
    b = batch.concatenate(inst)
    k = lattice.bond_stiffness_pmb(BULK_MODULUS, HORIZON_CELLS * DX)
    integ = pp.EulerCromerCUDA(DAMPING, dt=DT, precision="mixed")
    sim = batch.BatchedSimulation(b, integ, k)
    setup_s = time.perf_counter() - t0
    ms = time_steps(integ, steps, warmup, torch) / steps
    kernel_ms = time_kernel_launches(integ, 20, torch)
    alg = b.bonds * (4 + 8) + b.nnodes * B_NODE_VV
    out = {"bond_updates_per_s": b.bonds / (ms * 1e-3), "ms_per_step": ms,
           "kernel_ms": kernel_ms, "kernel": _kernel_name(integ),
           "algorithmic_bytes_per_launch": alg,
           "roofline_frac": _roofline_frac(alg, kernel_ms, peak),
           "nodes": b.nnodes, "bonds": b.bonds, "instances": len(inst),
           "timed_steps": steps, "setup_s": setup_s,
           "autotune_ms": integ.tuning,
           "tuned_vs_default": _tuning_summary(integ.tuning)}
    del integ, sim
    torch.cuda.empty_cache()
    return out


def variant_composite(torch, peak, ctx, steps=20, warmup=3):
    """The irregular composite, briefly: 1M Poisson-disk points, three bond
    types, trilinear damage, Velocity-Verlet, compensated force sums, faces
    pulled COMPOSITE_RATE per step.  Algorithmic bytes: neighbour index,
    bond type and regime (4 B each) per bond, 336 B per node."""
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300.pointset import composite
    t0 = time.perf_counter()
    w = composite(context=ctx)
    setup_s = time.perf_counter() - t0
    n = w["coords"].shape[0]
    bonds = int(w["family"].sum())
    integ = pp.VelocityVerletCUDA(DAMPING, dt=DT, precision="mixed",
                                  compensated=True, context=ctx)
    integ.build(n, 3, w["max_neigh"], w["coords"], w["volume"], w["family"],
                w["bc_types"], w["bc_values"], np.zeros((n, 3), dtype=np.intc),
                np.zeros((n, 3)), None, w["bond_types"], w["densities"])
    z = np.zeros((n, 3))
    integ.create_buffers(w["nlist"], w["n_neigh"], w["bond_stiffness"],
                         w["critical_stretch"], w["plus_cs"], z, z, z, z, z,
                         np.zeros(n), None, w["nregimes"], w["nbond_types"])
    ms = time_steps(integ, steps, warmup, torch, rate=COMPOSITE_RATE) / steps
    kernel_ms = time_kernel_launches(integ, 50, torch, rate=COMPOSITE_RATE)
    alg = bonds * (4 + 4 + 4) + n * B_NODE_VV
    out = {"bond_updates_per_s": bonds / (ms * 1e-3), "ms_per_step": ms,
           "kernel_ms": kernel_ms, "kernel": _kernel_name(integ),
           "algorithmic_bytes_per_launch": alg,
           "roofline_frac": _roofline_frac(alg, kernel_ms, peak),
           "nodes": n, "bonds": bonds, "max_neigh": w["max_neigh"],
           "timed_steps": steps, "setup_s": setup_s,
           "autotune_ms": integ.tuning,
           "tuned_vs_default": _tuning_summary(integ.tuning)}
    del integ
    torch.cuda.empty_cache()
    return out


def variant_adjoint(torch, passes=2, warmup=1):
    """One forward + checkpointed backward pass of the adjoint rollout
    (50x50x5 lattice, 500 binary64 Euler steps, checkpoint every 50, 100
    probe nodes); bond-updates count the forward, recomputed forward and
    reverse steps."""
    from probabilistic_peridynamics_gb300 import lattice
    from probabilistic_peridynamics_gb300.adjoint import (AdjointProblem,
                                                          rollout)
    nx, ny, nz, steps, every = 50, 50, 5, 500, 50
    coords = lattice.lattice_coords(nx, ny, nz, 1.0)
    family, nlist, _ = lattice.lattice_family(nx, ny, nz, HORIZON_CELLS)
    bc_types, bc_values = lattice.face_bcs(coords, 0)
    n = coords.shape[0]
    prob = AdjointProblem(coords, np.ones(n), nlist, bc_types, bc_values,
                          1e-9 * np.arange(1, steps + 1), 0.5)
    rng = np.random.default_rng(4)
    probes = torch.tensor(rng.choice(n, 100, replace=False), device="cuda")
    k0 = np.where(nlist != -1, 0.01 * rng.uniform(0.9, 1.1, nlist.shape),
                  0.0)
    k = torch.tensor(k0, dtype=torch.float32, device="cuda",
                     requires_grad=True)

    def one():
        k.grad = None
        u = rollout(k, 1.0, prob, steps, every)
        (u[probes] ** 2).sum().backward()

    for _ in range(warmup):
        one()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(passes):
        one()
    e1.record()
    e1.synchronize()
    ms = e0.elapsed_time(e1) / passes
    bonds = int(family.sum())
    del prob, k
    torch.cuda.empty_cache()
    return {"ms_per_pass": ms, "passes_per_s": 1e3 / ms,
            "bond_updates_per_s": bonds * steps * 3 / (ms * 1e-3),
            "nodes": n, "bonds": bonds, "steps": steps,
            "checkpoint_every": every, "arithmetic": "binary64"}


def e2e_simulate(w, torch):
    """Full 5000-step Model.simulate with host arrays in and out."""
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300.mesh import write_vtk
    tmp = tempfile.mkdtemp()
    mesh = os.path.join(tmp, "lattice.vtk")
    write_vtk(mesh, w["coords"], [])
    lo, hi = w["coords"][:, 0].min(), w["coords"][:, 0].max()

    def is_bnd(x):
        if x[0] <= lo + 1e-9:
            return [-1.0, None, None]
        if x[0] >= hi - 1e-9:
            return [1.0, None, None]
        return [None, None, None]

    integ = pp.VelocityVerletCUDA(DAMPING, dt=DT, precision="mixed")
    import warnings
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        model = pp.Model(mesh, integ, horizon=w["horizon"],
                         critical_stretch=S0, bond_stiffness=w["k"],
                         transfinite=1,
                         volume_total=float(w["volume"].sum()),
                         connectivity=(w["nlist"], w["n_neigh"]),
                         family=w["family"], dimensions=3,
                         density=np.full(w["nnodes"], DENSITY),
                         is_displacement_boundary=is_bnd)
    mags = PULL_RATE * np.arange(1, E2E_STEPS + 1)
    model.simulate(steps=20, displacement_bc_magnitudes=mags)  # warm-up
    # where the wall time goes: the integrator calls Model.simulate makes
    # (each already ends in, or is followed by, a synchronisation)
    parts = {}

    def timed(name):
        fn = getattr(integ, name)

        def call(*a, **k):
            t = time.perf_counter()
            try:
                return fn(*a, **k)
            finally:
                if name == "_run":
                    torch.cuda.synchronize()
                parts[name] = parts.get(name, 0.0) + time.perf_counter() - t
        setattr(integ, name, call)

    for name in ("create_buffers", "_run", "write"):
        timed(name)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    u, damage, (nlist, n_neigh), force, ud, _ = model.simulate(
        steps=E2E_STEPS, displacement_bc_magnitudes=mags)
    torch.cuda.synchronize()
    dt_s = time.perf_counter() - t0
    n = w["nnodes"]
    # create_buffers: nlist, n_neigh, u, ud, udd; per-segment magnitudes
    h2d = (w["nlist"].nbytes + w["n_neigh"].nbytes + 3 * n * 24
           + E2E_STEPS * 16)
    d2h = 5 * n * 24 + n * 8 + nlist.nbytes + n_neigh.nbytes
    return {"value": w["bonds"] * E2E_STEPS / dt_s, "unit": UNIT,
            "h2d_bytes_per_step": h2d / E2E_STEPS,
            "d2h_bytes_per_step": d2h / E2E_STEPS,
            "steps": E2E_STEPS, "wall_s": dt_s,
            "wall_parts_s": {"create_buffers": parts.get("create_buffers"),
                             "steps": parts.get("_run"),
                             "write": parts.get("write"),
                             "rest": dt_s - sum(parts.values())},
            "path": "Model.simulate (VelocityVerletCUDA, precision='mixed')"}


# --------------------------------------------------------------- CPU side
def reference_step_fn():
    """The reference's CPU Euler step, or None when it is not built."""
    try:
        from oracle import build_ref
        if not build_ref.available():
            build_ref.build(quiet=True)
        mod = build_ref.load()
    except Exception:  # noqa: BLE001 - any failure means "not available"
        return None
    return mod


def compact(nlist, family):
    width = int(family.max())
    out = np.ascontiguousarray(nlist[:, :width]).astype(np.intc)
    out[out == -1] = 0
    return out


#: Pseudo-time step of the reference's Euler update on the CPU samples.  The
#: reference CPU path has no Velocity-Verlet, and its Euler update
#: u += dt f is stable only for dt below 2 / lambda_max, lambda_max <=
#: 2 sum_j c vol / |xi_j| ~ 3e14 on this lattice: at larger dt displacements
#: grow, every bond breaks within a few steps and the sample stops doing
#: bond work.  At 1e-15 (dt lambda_max ~ 0.3) no bond breaks and each step
#: does the workload's bond work.
CPU_DT = 1e-15


def cpu_block(nx, ny=NY):
    """The reference CPU step on an nx x ny x 10 block of the lattice.

    :returns: (step(s) function, bonds per step, kind, cores, intact()
        function)
    """
    from probabilistic_peridynamics_gb300 import lattice
    mod = reference_step_fn()
    coords = lattice.lattice_coords(nx, ny, NZ, DX)
    # the C restatement takes rows of a power-of-two width
    family, nlist, _ = lattice.lattice_family(nx, ny, NZ, HORIZON_CELLS,
                                              pow2=mod is None)
    n = coords.shape[0]
    bonds = int(family.sum())
    k = lattice.bond_stiffness_pmb(BULK_MODULUS, HORIZON_CELLS * DX)
    bc_types, bc_values = lattice.face_bcs(coords, 0)
    vol = np.full(n, DX ** 3)
    fct = np.zeros((n, 3), dtype=np.intc)
    fcv = np.zeros((n, 3))
    u = np.zeros((n, 3))
    n_neigh = family.copy()
    # the same strain rate as the full plate: a block nx cells wide is
    # pulled (nx - 1)/(NX - 1) as fast
    rate = PULL_RATE * (nx - 1) / (NX - 1)
    if mod is not None:
        nl = compact(nlist, family)

        def step(s):
            mod.break_bonds(coords + u, coords, nl, n_neigh, S0)
            f = mod.bond_force(coords + u, coords, nl, n_neigh, vol, k, fcv,
                               fct, 0.0)
            mod.update_displacement(u, bc_values, bc_types, f, rate * s,
                                    CPU_DT)

        def intact():
            return int(n_neigh.sum())
        kind, cores = "reference", 1
    else:
        from oracle import cref
        st = cref.Stepper("euler", CPU_DT, coords, vol, family, nlist,
                          bc_types, bc_values, fct, fcv, k, S0)

        def step(s):
            st.step(rate * s, 0.0)

        def intact():
            return int((st.nlist != -1).sum())
        kind, cores = "port", os.cpu_count() or 1
    return step, bonds, kind, cores, intact


def cpu_sample(nx, budget_s, min_steps=1, max_steps=5, steps=None, ny=NY):
    """Time the reference CPU step on an nx x ny x 10 block of the lattice.

    :returns: (bond-updates/s, steps run, seconds, bonds per step, kind,
        cores, bonds broken during the sample)
    """
    step, bonds, kind, cores, intact = cpu_block(nx, ny)
    t0 = time.perf_counter()
    done = 0
    while True:
        step(done + 1)
        done += 1
        el = time.perf_counter() - t0
        if steps is not None:
            if done >= steps:
                break
        elif done >= max_steps or (el >= budget_s and done >= min_steps):
            break
    el = time.perf_counter() - t0
    return bonds * done / el, done, el, bonds, kind, cores, bonds - intact()


def host_cpu():
    """Model name and core count of the host, for the CPU lines."""
    model = None
    try:
        for line in pathlib.Path("/proc/cpuinfo").read_text().splitlines():
            key = line.split(":")[0].strip().lower()
            if key in ("model name", "cpu model", "hardware") and ":" in line:
                model = line.split(":", 1)[1].strip()
                break
    except OSError:
        pass
    if not model:
        import platform
        model = platform.processor() or platform.machine()
    return {"cpu": model, "host_cores": os.cpu_count()}


def cpu_baseline():
    rate, steps, el, bonds, kind, cores, broken = cpu_sample(NX,
                                                             budget_s=10.0)
    what = ("reference Cython Euler step (peripy/peridynamics.pyx break_bonds"
            " + bond_force + update_displacement)" if kind == "reference"
            else "C restatement of the OpenCL step (OpenMP)")
    return {"value": rate, "unit": UNIT, "cores": cores, "kind": kind,
            **host_cpu(),
            "sample": f"{steps} step(s) of the {what} on the full "
                      f"{NX}x{NY}x{NZ} lattice ({bonds} bonds/step, Euler "
                      f"dt {CPU_DT:g}, {broken} bonds broken), {el:.1f} s"}


def _reference_worker(nx, ny, warmup, steps, barrier, out):
    """One instance of the reference CPU step (a spawned process): its own
    block, the warm-up steps, then the timed steps started together with
    the other instances."""
    step, bonds, kind, cores, intact = cpu_block(nx, ny)
    for s in range(warmup):
        step(s + 1)
    barrier.wait()
    t0 = time.time()
    for s in range(steps):
        step(warmup + s + 1)
    t1 = time.time()
    out.put((bonds, steps, t0, t1, kind, cores,
             bonds - intact()))


def reference_arm(args):
    """The reference's own CPU step on the host cores.  The step is serial
    (no threads in the reference), so every core available to this process
    runs one instance of it on its own copy of the same block of the
    lattice, all timed over the same window: the rate is the bond-updates
    of all instances over that window."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import multiprocessing as mp
    total = args.steps + args.warmup
    try:
        workers = len(os.sched_getaffinity(0))
    except AttributeError:
        workers = os.cpu_count() or 1
    if reference_step_fn() is None:
        workers = 1  # the C port threads itself (OpenMP)
    # Size the block (4 x ny x 10 of the lattice) so that warm-up + timed
    # steps take about 90 s on one core; at most 50 x 200 x 10 per instance
    # (each instance holds its own block).
    probe_rate, *_ = cpu_sample(4, budget_s=0.5, min_steps=1, max_steps=3)
    per_step_bonds = probe_rate * 90.0 / max(total, 1)
    bonds_4xNY = 4 * NY * NZ * 107.0  # about 107 bonds per node in bulk
    nx, ny = 4, int(max(4, min(NY, NY * per_step_bonds / bonds_4xNY)))
    if per_step_bonds > bonds_4xNY:
        nx = int(max(4, min(50, 4 * per_step_bonds / bonds_4xNY)))
        ny = NY
    ctx = mp.get_context("spawn")
    barrier = ctx.Barrier(workers)
    out = ctx.Queue()
    procs = [ctx.Process(target=_reference_worker,
                         args=(nx, ny, args.warmup, args.steps, barrier, out))
             for _ in range(workers)]
    for p in procs:
        p.start()
    res = [out.get() for _ in procs]
    for p in procs:
        p.join()
    bonds = res[0][0]
    steps = args.steps
    t0 = min(r[2] for r in res)
    t1 = max(r[3] for r in res)
    el = t1 - t0
    rate = sum(r[0] * r[1] for r in res) / el
    kind = res[0][4]
    broken = res[0][6]
    what = ("the reference CPU step (Cython break_bonds + bond_force + "
            "update_displacement)" if kind == "reference" else
            "C restatement of the OpenCL step")
    sample = (f"each step: {what}, {workers} instances at once (one per "
              f"core: the reference step is serial), each on a {nx}x{ny}x"
              f"{NZ} block of the lattice ({bonds} bonds, Euler dt "
              f"{CPU_DT:g}, {broken} bonds broken over the run)")
    cores = workers
    line = {
        "impl": "reference", "metric": METRIC, "value": rate, "unit": UNIT,
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * el / max(steps, 1), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic",
        "config": {"workload": WORKLOAD, "sample": sample,
                   "integrator": "Euler (the reference CPU path has no "
                                 "Velocity-Verlet)"},
        "cpu_baseline": {"value": rate, "unit": UNIT, "cores": cores,
                         "kind": kind, **host_cpu(), "sample": sample},
        "e2e": {"value": rate, "unit": UNIT, "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# -------------------------------------------------------------------- main
def load_peaks():
    try:
        return json.loads((ROOT / "MEASURED_PEAKS.json").read_text())
    except (OSError, ValueError):
        return None


def load_traffic(kernel):
    """DRAM bytes per launch of ``kernel`` on the plate from the committed
    ncu summary (``profiles/<kernel>_vv_200x200x10_traffic.txt``: a
    ``dram_bytes_per_launch N`` line)."""
    for p in sorted((ROOT / "profiles").glob(f"{kernel}_*traffic*.txt")):
        for line in p.read_text().splitlines():
            if line.startswith("dram_bytes_per_launch"):
                try:
                    return float(line.split()[1])
                except (IndexError, ValueError):
                    pass
    return None


def batched_main(args):
    """64 uneven UQ instances in one persistent launch per step."""
    import torch
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import batch, lattice
    t0 = time.perf_counter()
    inst = batch.uq_instances(count=64, seed=2024, dx=DX)
    b = batch.concatenate(inst)
    setup_s = time.perf_counter() - t0
    k = lattice.bond_stiffness_pmb(BULK_MODULUS, HORIZON_CELLS * DX)
    integ = pp.EulerCromerCUDA(DAMPING, dt=DT, precision="mixed")
    sim = batch.BatchedSimulation(b, integ, k)
    steps, warmup = args.steps, args.warmup
    ms = time_steps(integ, steps, warmup, torch)
    value = b.bonds * steps / (ms * 1e-3)
    kernel_ms = time_kernel_launches(integ, 50, torch)
    alg = b.bonds * (4 + 8) + b.nnodes * B_NODE_VV
    peaks = load_peaks()
    peak = float(peaks["hbm_gbs"]) if peaks else 6800.0
    achieved = alg / (kernel_ms * 1e-3) / 1e9
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": 1,
        "steps": steps, "warmup": warmup, "ms_per_step": ms / steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32", "data": "synthetic",
        "config": {"workload": "batched UQ: 64 instances nx,ny~U{60..200}, "
                               "nz=5, Euler-Cromer, lognormal s0, "
                               "U(0.9,1.1) bond noise",
                   "nodes": b.nnodes, "bonds": b.bonds,
                   "instances": len(inst), "setup_s": setup_s,
                   "tile_shape_autotune_ms": integ.tuning,
                   "variant": int(integ._fargs.variant)},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak,
                     "unit": "GB/s", "frac": achieved / peak,
                     "algorithmic_bytes_per_launch": alg,
                     "kernel_ms": kernel_ms},
        "gpu_launches": steps + (steps // 16 + 1 if steps >= 32 else 0),
    }
    print(json.dumps(line), flush=True)


COMPOSITE_RATE = 5e-7


def composite_main(args):
    """The irregular composite: 1M Poisson-disk points in 2.0 x 1.0 x 0.1,
    horizon 0.012, bond types 0/1/2 (K = 1e9, 3e9, harmonic-mean interface),
    trilinear damage (0.004, 0.006, 0.01), Velocity-Verlet with density
    2400, damping 2.5e6, dt 1e-6, x faces pulled 5e-7 per step; mixed step
    with compensated force sums, its error against the FP64 step after
    ``--accuracy-steps`` steps with and without compensation, beside the
    error of an FP64 run whose initial velocities are perturbed by
    3e-12 m/s (through fracture the problem amplifies any perturbation)."""
    import torch
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300.pointset import composite
    from probabilistic_peridynamics_gb300.integrators import CUDAContext
    from probabilistic_peridynamics_gb300.model import (build_family,
                                                        neighbour_pairs)
    from probabilistic_peridynamics_gb300.neighbours import neighbour_family
    ctx = CUDAContext(0)
    t0 = time.perf_counter()
    w = composite(context=ctx)
    setup_s = time.perf_counter() - t0
    n = w["coords"].shape[0]
    bonds = int(w["family"].sum())
    # neighbour families of the 1M points: GPU cell search vs host KD-tree
    neighbour_family(w["coords"], w["horizon"], ctx)  # warm
    t0 = time.perf_counter()
    fam_g, nl_g, _ = neighbour_family(w["coords"], w["horizon"], ctx)
    gpu_s = time.perf_counter() - t0
    t0 = time.perf_counter()
    fam_h, nl_h, _ = build_family(n, neighbour_pairs(w["coords"],
                                                     w["horizon"]))
    host_s = time.perf_counter() - t0
    neighbours = {"gpu_s": gpu_s, "host_kdtree_s": host_s,
                  "identical": bool(np.array_equal(fam_g, fam_h) and
                                    np.array_equal(nl_g, nl_h))}
    del nl_g, nl_h

    def make(precision, compensated=False, ud0=None):
        integ = pp.VelocityVerletCUDA(DAMPING, dt=DT, precision=precision,
                                      compensated=compensated)
        integ.build(n, 3, w["max_neigh"], w["coords"], w["volume"],
                    w["family"], w["bc_types"], w["bc_values"],
                    np.zeros((n, 3), dtype=np.intc), np.zeros((n, 3)), None,
                    w["bond_types"], w["densities"])
        z = np.zeros((n, 3))
        integ.create_buffers(w["nlist"], w["n_neigh"], w["bond_stiffness"],
                             w["critical_stretch"], w["plus_cs"], z,
                             z if ud0 is None else ud0, z, z, z, np.zeros(n),
                             None, w["nregimes"], w["nbond_types"])
        return integ

    integ = make("mixed", compensated=True)
    clocks = ClockSampler(0)
    clocks.start()
    ms = time_steps(integ, args.steps, args.warmup, torch,
                    rate=COMPOSITE_RATE)
    clk = clocks.stop()
    kernel_ms = time_kernel_launches(integ, 100, torch, rate=COMPOSITE_RATE)
    tuning, variant = integ.tuning, int(integ._fargs.variant)
    del integ
    torch.cuda.empty_cache()
    acc = None
    if args.accuracy_steps:
        steps = args.accuracy_steps
        mags = COMPOSITE_RATE * np.arange(1, steps + 1)
        res = {}
        # the FP64 run from initial velocities perturbed by 3e-12 m/s shows
        # how far the problem itself carries a perturbation
        pert = 3e-12 * np.random.default_rng(0).standard_normal((n, 3))
        for name, prec, comp, ud0 in (
                ("fp64", "float64", False, None),
                ("fp64_perturbed", "float64", False, pert),
                ("mixed", "mixed", False, None),
                ("mixed_compensated", "mixed", True, None)):
            it = make(prec, comp, ud0)
            it._run(mags, np.zeros(steps), 0, steps)
            z = [np.zeros((n, 3)) for _ in range(5)]
            res[name] = it.write(*z, np.zeros(n), w["nlist"].copy(),
                                 w["n_neigh"].copy())
            del it
            torch.cuda.empty_cache()
        u64, nl64 = res["fp64"][0], res["fp64"][6]
        acc = {"steps": steps,
               "bonds_broken_fp64": int((w["nlist"] != -1).sum() -
                                        (nl64 != -1).sum()),
               "max_abs_u": float(np.abs(u64).max())}
        for name in ("fp64_perturbed", "mixed", "mixed_compensated"):
            u = res[name][0]
            acc[name] = {
                "disp_rel_err_vs_fp64": float(np.abs(u - u64).max() /
                                              np.abs(u64).max()),
                "mask_flips_vs_fp64": int((res[name][6] != nl64).sum()),
                "bonds_broken": int((w["nlist"] != -1).sum() -
                                    (res[name][6] != -1).sum())}
    peaks = load_peaks()
    peak = float(peaks["hbm_gbs"]) if peaks else 6800.0
    # int32 nlist + bond_types + regimes per bond; VV node bytes
    alg = bonds * (4 + 4 + 4) + n * B_NODE_VV
    achieved = alg / (kernel_ms * 1e-3) / 1e9
    line = {
        "metric": METRIC, "value": bonds * args.steps / (ms * 1e-3),
        "unit": UNIT, "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32", "data": "synthetic",
        "config": {"workload": "irregular composite: 1M Poisson-disk points "
                               "in 2.0x1.0x0.1, 3 bond types, trilinear "
                               "damage, Velocity-Verlet",
                   "nodes": n, "bonds": bonds, "max_neigh": w["max_neigh"],
                   "setup_s": setup_s, "neighbour_build": neighbours,
                   "pull_rate": COMPOSITE_RATE,
                   "precision": "mixed, compensated force sums",
                   "tile_shape_autotune_ms": tuning, "variant": variant},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak,
                     "unit": "GB/s", "frac": achieved / peak,
                     "algorithmic_bytes_per_launch": alg,
                     "kernel_ms": kernel_ms},
        "gpu_launches": args.steps + (args.steps // 16 + 1
                                      if args.steps >= 32 else 0),
        "clocks": clk, "accuracy": acc,
    }
    print(json.dumps(line), flush=True)


def adjoint_main(args):
    """Gradient of a displacement loss through the Euler rollout: the
    50x50x5 lattice (dx 1, horizon 3.015, per-bond stiffness 0.01 U(0.9,1.1)
    as a float32 parameter), faces pulled 1e-9 per step, dt 0.5, 500 steps,
    checkpoint every 50, loss = sum of squared displacements of 100 seeded
    probe nodes.  One step of this line = one forward + backward pass."""
    import torch
    from probabilistic_peridynamics_gb300 import lattice
    from probabilistic_peridynamics_gb300.adjoint import (AdjointProblem,
                                                          rollout)
    nx, ny, nz, steps, every = 50, 50, 5, 500, 50
    coords = lattice.lattice_coords(nx, ny, nz, 1.0)
    family, nlist, _ = lattice.lattice_family(nx, ny, nz, HORIZON_CELLS)
    bc_types, bc_values = lattice.face_bcs(coords, 0)
    n = coords.shape[0]
    prob = AdjointProblem(coords, np.ones(n), nlist, bc_types, bc_values,
                          1e-9 * np.arange(1, steps + 1), 0.5)
    rng = np.random.default_rng(4)
    probes = torch.tensor(rng.choice(n, 100, replace=False), device="cuda")
    k0 = np.where(nlist != -1, 0.01 * rng.uniform(0.9, 1.1, nlist.shape),
                  0.0)
    k = torch.tensor(k0, dtype=torch.float32, device="cuda",
                     requires_grad=True)

    def one():
        k.grad = None
        u = rollout(k, 1.0, prob, steps, every)
        (u[probes] ** 2).sum().backward()

    for _ in range(args.warmup):
        one()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.steps):
        one()
    e1.record()
    e1.synchronize()
    ms = e0.elapsed_time(e1) / args.steps
    bonds = int(family.sum())
    # forward steps + recomputed forward steps + reverse steps per pass
    updates = bonds * steps * 3
    line = {
        "metric": "adjoint passes/s (forward + checkpointed backward)",
        "value": 1e3 / ms, "unit": "passes/s", "n_gpus": 1,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f64", "data": "synthetic",
        "config": {"workload": "adjoint: 50x50x5 lattice, 500 Euler steps, "
                               "checkpoint every 50, 100 probes",
                   "nodes": n, "bonds": bonds,
                   "bond_updates_per_s": updates / (ms * 1e-3)},
    }
    print(json.dumps(line), flush=True)


def writes_main(args):
    """Model.simulate on the 200x200x10 plate with a write every 500 of
    5000 Velocity-Verlet steps (mixed precision): mesh files of u and damage
    plus the recorded sums, with one tip type (the x dof of the pulled
    x-max face).  Timed twice through the public API: with the write-step
    sums on the device (only u and damage come back) and with the host path
    that copies all eight state arrays back at every write (the reference's
    Integrator.write), both writing the same files and data."""
    import torch
    import warnings
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300.mesh import write_vtk
    w = build_workload()
    steps, every = E2E_STEPS, 500
    tmp = tempfile.mkdtemp()
    mesh = os.path.join(tmp, "lattice.vtk")
    write_vtk(mesh, w["coords"], [])
    lo, hi = w["coords"][:, 0].min(), w["coords"][:, 0].max()

    def is_bnd(x):
        if x[0] <= lo + 1e-9:
            return [-1.0, None, None]
        if x[0] >= hi - 1e-9:
            return [1.0, None, None]
        return [None, None, None]

    def is_tip(x):
        return ["pulled", None, None] if x[0] >= hi - 1e-9 else \
            [None, None, None]

    class HostWrites(pp.VelocityVerletCUDA):
        write_sums = None

    mags = PULL_RATE * np.arange(1, steps + 1)
    out = {}
    for name, cls in (("device_sums", pp.VelocityVerletCUDA),
                      ("host_copies", HostWrites)):
        integ = cls(DAMPING, dt=DT, precision="mixed")
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")
            model = pp.Model(mesh, integ, horizon=w["horizon"],
                             critical_stretch=S0, bond_stiffness=w["k"],
                             transfinite=1,
                             volume_total=float(w["volume"].sum()),
                             connectivity=(w["nlist"], w["n_neigh"]),
                             family=w["family"], dimensions=3,
                             density=np.full(w["nnodes"], DENSITY),
                             is_displacement_boundary=is_bnd, is_tip=is_tip)
        path = pathlib.Path(tmp) / name
        path.mkdir()
        model.simulate(steps=20, displacement_bc_magnitudes=mags, write=10,
                       write_path=path)  # warm-up
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        res = model.simulate(steps=steps, displacement_bc_magnitudes=mags,
                             write=every, write_path=path)
        torch.cuda.synchronize()
        out[name] = (time.perf_counter() - t0, res[5])
        del model, integ
        torch.cuda.empty_cache()
    dev_s, dev_data = out["device_sums"]
    host_s, host_data = out["host_copies"]
    same = all(np.array_equal(dev_data[k][f], host_data[k][f])
               for k in host_data for f in host_data[k])
    n = w["nnodes"]
    nwrites = steps // every
    line = {
        "metric": "bond-updates/s through Model.simulate with writes",
        "value": w["bonds"] * steps / dev_s, "unit": UNIT, "n_gpus": 1,
        "steps": steps, "warmup": 20, "ms_per_step": 1e3 * dev_s / steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32+f64", "data": "synthetic",
        "config": {"workload": WORKLOAD + f"; write every {every} steps "
                               "(mesh file + recorded sums), one tip type",
                   "writes": nwrites, "nodes": n, "bonds": w["bonds"]},
        "variants": {
            "device_sums": {"wall_s": dev_s,
                            "d2h_bytes_per_write": n * 24 + n * 8},
            "host_copies": {"wall_s": host_s,
                            "d2h_bytes_per_write":
                                5 * n * 24 + n * 8 + w["nlist"].nbytes
                                + w["n_neigh"].nbytes,
                            "value": w["bonds"] * steps / host_s}},
        "data_identical": bool(same),
    }
    print(json.dumps(line), flush=True)


def setup_main(args):
    """Model set-up of the 200x200x10 plate on the GPU: neighbour families
    (cell search) and the plane crack (30,940 pairs, pp_create_crack), each
    timed on device-resident arrays (CUDA events, median of --steps runs
    after --warmup) and through the host-array entry points; beside them
    the host search (scipy cKDTree pairs assembled into rows) and the
    reference's own compiled create_crack on one core, all on the same
    arrays and checked equal."""
    import torch
    from probabilistic_peridynamics_gb300 import lattice
    from probabilistic_peridynamics_gb300.integrators import CUDAContext
    from probabilistic_peridynamics_gb300.model import (build_family,
                                                        neighbour_pairs)
    from probabilistic_peridynamics_gb300.neighbours import (
        crack_device, create_crack, neighbour_family)
    ctx = CUDAContext(0)
    coords = lattice.lattice_coords(NX, NY, NZ, DX)
    horizon = HORIZON_CELLS * DX
    family, nlist, _ = neighbour_family(coords, horizon, ctx)
    t0 = time.perf_counter()
    family, nlist, _ = neighbour_family(coords, horizon, ctx)
    nb_gpu_s = time.perf_counter() - t0
    t0 = time.perf_counter()
    fam_h, nl_h, _ = build_family(coords.shape[0],
                                  neighbour_pairs(coords, horizon))
    nb_host_s = time.perf_counter() - t0
    same_rows = bool(np.array_equal(family, fam_h)
                     and np.array_equal(nlist, nl_h))
    n_neigh = family.copy()
    pairs = np.ascontiguousarray(
        lattice.plane_crack_pairs(coords, nlist, n_neigh, 0.5, 0.25),
        dtype=np.intc)
    dev = ctx.device
    with ctx.on_stream():
        nl_d = torch.as_tensor(nlist, device=dev)
        nn_d = torch.as_tensor(n_neigh, device=dev)
        c_d = torch.as_tensor(pairs, device=dev)
        times = []
        for k in range(max(args.warmup, 1) + max(args.steps, 1)):
            x, y = nl_d.clone(), nn_d.clone()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(ctx.stream)
            crack_device(c_d, x, y, ctx)
            e1.record(ctx.stream)
            e1.synchronize()
            if k >= max(args.warmup, 1):
                times.append(e0.elapsed_time(e1))
    crack_dev_ms = statistics.median(times)
    got_nl, got_nn = nlist.copy(), n_neigh.copy()
    t0 = time.perf_counter()
    create_crack(pairs, got_nl, got_nn, ctx)
    crack_host_arrays_s = time.perf_counter() - t0
    same_dev = bool(np.array_equal(x.cpu().numpy(), got_nl))
    ref = reference_step_fn()
    ref_s = None
    same_ref = None
    if ref is not None:
        from oracle import build_ref
        ref_crack = build_ref.load("create_crack").create_crack
        r_nl, r_nn = nlist.copy(), n_neigh.copy()
        t0 = time.perf_counter()
        ref_crack(pairs, r_nl, r_nn)
        ref_s = time.perf_counter() - t0
        same_ref = bool(np.array_equal(r_nl, got_nl)
                        and np.array_equal(r_nn, got_nn))
    line = {
        "metric": "initial-crack time on device-resident arrays",
        "value": crack_dev_ms, "unit": "ms", "n_gpus": 1,
        "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": crack_dev_ms, "higher_is_better": False,
        "scaling": "weak", "vs_baseline": None, "dtype": "int32",
        "data": "synthetic",
        "config": {"workload": "set-up of the 200x200x10 lattice "
                               "(400k nodes): neighbour families and the "
                               "plane crack x = 0.5, y < 0.25",
                   "crack_pairs": int(len(pairs)),
                   "bonds": int(family.sum())},
        "crack": {"device_ms": crack_dev_ms,
                  "host_arrays_s": crack_host_arrays_s,
                  "same_as_host_array_path": same_dev,
                  "reference_compiled_s": ref_s,
                  "same_as_reference": same_ref},
        "neighbours": {"gpu_s": nb_gpu_s, "host_kdtree_s": nb_host_s,
                       "same_rows": same_rows},
        "cpu_baseline": ({"value": ref_s * 1e3, "unit": "ms", "cores": 1,
                          "kind": "reference",
                          "sample": "the reference's compiled "
                                    "create_crack on the same crack list"}
                         if ref_s is not None else None),
    }
    print(json.dumps(line), flush=True)


def main():
    args = parse_args()
    if args.profile:
        profile_case(args.profile)
        return
    if args.impl == "reference":
        reference_arm(args)
        return
    if args.workload == "batched":
        batched_main(args)
        return
    if args.workload == "composite":
        composite_main(args)
        return
    if args.workload == "adjoint":
        adjoint_main(args)
        return
    if args.workload == "writes":
        writes_main(args)
        return
    if args.workload == "setup":
        setup_main(args)
        return
    import torch
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch.distributed as tdist
        torch.cuda.set_device(local)
        tdist.init_process_group("nccl")
        dist = tdist
    from probabilistic_peridynamics_gb300.integrators import CUDAContext
    ctx = CUDAContext(local)
    w = build_workload()
    integ = make_integrator(w, "mixed", True, context=ctx)
    # clocks sampled from the warm-up through the per-launch timing (the
    # timed region alone can be shorter than one 200 ms sample)
    clocks = ClockSampler(local)
    clocks.start()
    ms = time_steps(integ, args.steps, args.warmup, torch, dist)
    ms = job_time_ms(ms, dist, torch, "cuda")
    ms_per_step = ms / args.steps
    value = job_throughput(world, w["bonds"], args.steps, ms)
    kernel_ms = time_kernel_launches(integ, 200, torch)
    # about a second more of the same steps under the sampler, so that the
    # clocks are seen under sustained load (not timed)
    burst = max(1, int(1000.0 / max(ms_per_step, 1e-3)))
    time_steps(integ, burst, 0, torch)
    clk = clocks.stop()
    clk["window"] = ("warm-up, timed steps, 200 timed launches and "
                     f"{burst} further steps (untimed)")
    tuning = integ.tuning
    variant = int(integ._fargs.variant)
    kernel = "k_tiled" if integ.tiling is not None else "k_mixed"
    tiling_stats = integ.tiling.stats() if integ.tiling is not None else None
    launches = args.steps + (args.steps // 16 + 1
                             if args.steps >= 32 else 0)
    del integ
    torch.cuda.empty_cache()
    if rank != 0:
        if dist is not None:
            dist.barrier()
        return

    peaks = load_peaks()
    peak = float(peaks["hbm_gbs"]) if peaks else 6800.0
    alg_bytes = w["bonds"] * B_BOND + w["nnodes"] * B_NODE_VV
    achieved = alg_bytes / (kernel_ms * 1e-3) / 1e9
    traffic = load_traffic(kernel)

    variants = {"fused_mixed": {"bond_updates_per_s": value,
                                "ms_per_step": ms_per_step,
                                "kernel_ms": kernel_ms,
                                "autotune_ms": tuning,
                                "tuned_vs_default": _tuning_summary(tuning),
                                "variant": variant, "kernel": kernel,
                                "tiling": tiling_stats}}
    for name, precision, fused in (("plain_fp64", "float64", False),
                                   ("fused_fp64", "float64", True)):
        it = make_integrator(w, precision, fused, context=ctx)
        if fused:
            ms64 = time_steps(it, args.fp64_steps, 2, torch) / args.fp64_steps
        else:
            ms64 = time_plain_steps(it, args.fp64_steps, 2, torch)
        variants[name] = {"bond_updates_per_s": w["bonds"] / (ms64 * 1e-3),
                          "ms_per_step": ms64}
        del it
        torch.cuda.empty_cache()
    variants["speedup_mixed_vs_plain_fp64"] = (
        value / variants["plain_fp64"]["bond_updates_per_s"])
    variants["euler_cython_gpu"] = time_cython_euler(w, args.fp64_steps,
                                                     torch)

    variants["fused_mixed_fracture"] = time_fracture(w, 20, torch, ctx)
    if not args.no_variants:
        variants["batched_uq"] = variant_batched(torch, peak)
        variants["composite"] = variant_composite(torch, peak, ctx)
        variants["adjoint"] = variant_adjoint(torch)
    acc = accuracy(w, args.accuracy_steps, torch) if args.accuracy_steps \
        else None
    acc_fracture = accuracy_fracture(w, torch)
    e2e = None if args.no_e2e else e2e_simulate(w, torch)
    cpu = None if args.no_cpu else cpu_baseline()

    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": ms_per_step, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic",
        "config": {"workload": WORKLOAD, "nodes": w["nnodes"],
                   "bonds": w["bonds"], "max_neigh": w["max_neigh"],
                   "crack_pairs": w["crack_pairs"], "dt": DT,
                   "integrator": "Velocity-Verlet", "density": DENSITY,
                   "damping": DAMPING, "precision": "mixed (FP32 bonds, "
                   "exact FP64 stretch test, double-float state)",
                   "l2": "inputs larger than L2 (204.8 MB neighbour list "
                         "streamed per step), no flush",
                   "parallelism": "replicas" if world > 1 else "single"},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak,
                     "unit": "GB/s", "frac": achieved / peak,
                     "traffic": traffic,
                     "algorithmic_bytes_per_launch": alg_bytes,
                     "kernel": kernel,
                     "kernel_ms": kernel_ms,
                     "peak_source": ("measured" if peaks else "fallback")},
        "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": launches,
        "clocks": clk, "variants": variants, "accuracy": acc,
        "accuracy_fracture": acc_fracture,
    }
    print(json.dumps(line), flush=True)
    if dist is not None:
        dist.barrier()


if __name__ == "__main__":
    main()
