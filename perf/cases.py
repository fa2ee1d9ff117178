"""Performance cases of rfx_b200: what a program asks of it, with inputs, work and a 64-bit answer for each.

Every case is a scene (grid, materials, sources, monitors) built from a seed and one public way of running it:

  run        rfx_b200.run: host arrays in, traces, monitors and fields out (a closed or an absorbing box, a lumped
             port, an NTFF box with the far-field transform)
  nonuniform rfx_b200.run_nonuniform: the graded lane with a PEC sheet and a DFT plane
  decay      rfx_b200.run_until_decay: chunks of steps with an energy check between them
  steps      a resident plan restarted from given fields and advanced (the loop of a program that keeps its plan)
  adjoint    AdjointRunner / FDTDFunction: probe and DFT objectives, gradients of eps_r over a region and of the sources
  sweep      Sweep: forward and adjoint of many simulations of uneven size in one batch

The grids are those of rfx_b200/workloads.py, the tests' scenes and generic ones around them; step counts are cut so
that a pass stays within a fraction of a second.  ``exact`` marches the same scene in plain float64 torch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import rfx_b200
from rfx_b200.adjoint import AdjointRunner, FDTDFunction
from rfx_b200.batch import Sweep, SweepInstance
from rfx_b200.simulation import prepare_device_run

C0 = 299_792_458.0
EPS_0 = 8.8541878128e-12
MU_0 = 1.25663706212e-6
COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")


# ---------------------------------------------------------------------------
# the cases


def listed():
    return [
        # the README quick start: a small dielectric scene run once from host arrays, final fields wanted
        dict(name="quickstart_run", how="run", nx=87, ny=47, nz=42, ncp=8, dx=2e-3, f0=3e9, steps=1200, probes=1,
             state=True),
        # one frequency sweep of a small lumped-port structure (tests/scenarios.py small_uniform's grid): the
        # smallest call that is made in numbers, where latency and launches count
        dict(name="lumped_port_run", how="run", nx=43, ny=37, nz=33, ncp=6, dx=1e-3, f0=12e9, steps=400, probes=2,
             port=True, state=False),
        # an antenna run: NTFF box, flux monitor and the far field of it
        dict(name="antenna_run", how="run", nx=93, ny=101, nz=77, ncp=8, dx=1e-3, f0=9e9, steps=240, probes=1,
             ntff=3, flux=4, state=False),
        # the reference's own throughput benchmark (closed PEC box, no CPML) as a whole call
        dict(name="pec_benchmark_run", how="run", nx=257, ny=257, nz=257, ncp=0, dx=1e-3, f0=5e9, steps=400, probes=1,
             vacuum=True, state=False),
        # a run until the energy has decayed, checked every 50 steps (or until the cap: with the scene, after 250 to 400)
        dict(name="decay_run", how="decay", nx=61, ny=52, nz=49, ncp=8, dx=1e-3, f0=12e9, steps=400, probes=1),
        # the graded-lane configuration: CPML 12, PEC sheet, 8-frequency DFT plane
        dict(name="graded_run", how="nonuniform", nx=217, ny=217, nz=121, ncp=12, dx=5e-4, f0=20e9, steps=300,
             probes=4, dft=8, sheet=True, state=True),
        # the large uniform configuration (277^3, CPML 10, 8 probes, 16-frequency DFT plane), resident plan
        dict(name="uniform_277_steps", how="steps", nx=277, ny=277, nz=277, ncp=10, dx=1e-3, f0=10e9, steps=60,
             probes=8, dft=16),
        # odd sizes on every axis, per-cell mu_r, a PEC block, open y faces: the ordinary plan of a ragged scene
        dict(name="ragged_steps", how="steps", nx=131, ny=147, nz=103, ncp=8, dx=1e-3, f0=10e9, steps=60, probes=5,
             axes="xz", mu=True, sheet=True),
        # the largest grid: 513^3 closed box, resident plan
        dict(name="pec_513_steps", how="steps", nx=513, ny=513, nz=513, ncp=0, dx=1e-3, f0=5e9, steps=40, probes=1),
        # inverse design with checkpoints every 64 steps and segment recompute (the adjoint configuration, a
        # ragged last segment), gradients of a probe objective
        dict(name="adjoint_checkpointed", how="adjoint", nx=221, ny=141, nz=69, ncp=10, dx=5e-4, f0=15e9, steps=150,
             probes=4, box=64, every=64),
        # the autograd face in history mode: probe traces and a DFT plane, gradients of both inputs
        dict(name="adjoint_autograd", how="adjoint", nx=97, ny=83, nz=109, ncp=8, dx=1e-3, f0=10e9, steps=200,
             probes=3, box=16, dft=2, every=0),
        # a design sweep of uneven instances, forward + adjoint in one batch (the headline workload's size range)
        dict(name="sweep", how="sweep", n_inst=20, n_lo=64, n_hi=160, ncp=8, dx=5e-4, f0=12e9, steps=40),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    how = rng.choice(["run", "run", "decay", "nonuniform", "steps", "steps", "adjoint", "sweep"])
    ncp = rng.choice([0, 6, 8, 10, 12]) if how in ("run", "steps") else rng.choice([6, 8, 10, 12])
    f0 = rng.choice([5e9, 8e9, 10e9, 12e9])
    if how == "sweep":
        lo = rng.randint(20, 90)
        return dict(how=how, n_inst=rng.randint(2, 12), n_lo=lo, n_hi=lo + rng.randint(6, 50), ncp=8, dx=5e-4, f0=f0,
                    steps=rng.randint(30, 60))
    hi = {"run": 190, "decay": 90, "nonuniform": 200, "steps": 290, "adjoint": 140}[how]
    lo = max(28, 2 * ncp + 14)
    d = dict(how=how, nx=log(lo, hi), ny=log(lo, hi), nz=log(lo, hi), ncp=ncp, dx=1e-3, f0=f0, probes=rng.randint(1, 6))
    d["steps"] = {"run": 200, "decay": 360, "nonuniform": 150, "steps": 40, "adjoint": 100}[how] + rng.randint(0, 25)
    if how == "run":
        d["state"] = rng.random() < 0.5
        d["port"] = rng.random() < 0.3
        if rng.random() < 0.4:
            d["ntff"] = rng.randint(1, 3)
        if rng.random() < 0.4:
            d["flux"] = rng.randint(1, 5)
    if how in ("run", "nonuniform", "steps", "adjoint") and rng.random() < 0.5:
        d["dft"] = rng.randint(1, 12)
    if how in ("nonuniform", "steps", "run") and rng.random() < 0.5:
        d["sheet"] = True
    if how == "steps":
        d["mu"] = rng.random() < 0.25
        if ncp:
            d["axes"] = rng.choice(["xyz", "xyz", "xyz", "xy", "z", "yz"])
    if how == "adjoint":
        d["box"] = rng.randint(4, 12)
        d["every"] = rng.choice([0, 0, 24, 50])
        d["dx"] = 5e-4
    return d


def work(case):
    """Bytes of one pass: per step the six fields read and written and ca, cb read (56 B a cell), every CPML psi
    entry read and written (8 B), the accumulators of the monitors read and written; a pass with gradients marches
    once forward and once back, with checkpoints once more forward."""
    if case["how"] == "sweep":
        b = f = 0.0
        for n in _sweep_sizes(case):
            w = work(dict(case, how="steps", nx=n, ny=n, nz=n))
            b, f = b + 2 * w["bytes"] + case["steps"] * 40 * 512, f + 2 * w["flops"]
        return dict(bytes=b, flops=f)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ncp, axes, steps = case["ncp"], case.get("axes", "xyz"), case["steps"]
    cells = nx * ny * nz
    cross = dict(x=ny * nz, y=nx * nz, z=nx * ny)
    psi = sum(8 * ncp * cross[a] for a in axes) if ncp else 0
    per = 56 * cells + 8 * psi + 16 * case.get("dft", 0) * nx * ny
    if case.get("mu"):
        per += 4 * cells
    if case["how"] == "decay":
        steps *= 0.75        # it stops between 60 % of the cap and the cap
    flops = steps * (36.0 * cells + 6.0 * psi)
    if case.get("ntff"):
        lo, hi = _ntff_box(case)
        d = [h - q for q, h in zip(lo, hi)]
        faces = 2 * (d[0] * d[1] + d[1] * d[2] + d[0] * d[2])
        per += faces * 4 * 16 * case["ntff"]
        flops += faces * case["ntff"] * len(_angles()[0]) * len(_angles()[1]) * 60.0
    if case.get("flux"):
        per += 4 * 32 * case["flux"] * (ny - 2 * ncp) * (nz - 2 * ncp)
    b = float(steps) * per
    if case["how"] == "adjoint":
        b = b * (3 if case["every"] else 2) + steps * 40.0 * 2 * case["box"] ** 2
        flops *= 3 if case["every"] else 2
    return dict(bytes=b, flops=flops)


def tolerance(case):
    """float32 marches: about four times what the path measures against ``exact`` on an output (its coefficients and
    phase tables are float32 as well): resident steps 6e-7, the sweep's gradients 1e-6, whole runs 6e-5 (the smallest
    field component), gradients through an absorber 9e-5, the remains of a field that has decayed 4.5e-4."""
    return {"rel": {"steps": 4e-6, "sweep": 1e-5, "run": 3e-4, "nonuniform": 3e-4, "adjoint": 4e-4, "decay": 2e-3}[case["how"]]}


# ---------------------------------------------------------------------------
# scenes (numpy, from the seed alone)


class _Scene:
    pass


def _pulse(f0, steps, dt, amp, start=2.2):
    """Differentiated Gaussian, about as wide as the workloads' (bandwidth 0.8), ``start`` widths after the first step."""
    tau = 1.0 / (f0 * 0.8 * math.pi)
    a = (np.arange(steps) * dt - start * tau) / tau
    return (amp * -2.0 * a * np.exp(-a * a)).astype(np.float32)


def _carrier(f0, steps, dt, amp):
    """A carrier ramped up over a period and held to the last step, so that the final fields are a live field."""
    t = np.arange(steps) * dt * f0
    return (amp * (1.0 - np.exp(-t * t)) * np.sin(2.0 * math.pi * t)).astype(np.float32)


def _scene(case, seed):
    rng = np.random.default_rng([int(seed), 7])
    s = _Scene()
    s.case, s.steps, s.dx = case, case["steps"], case["dx"]
    s.shape = (case["nx"], case["ny"], case["nz"])
    s.ncp = case["ncp"]
    s.axes = case.get("axes", "xyz") if s.ncp else ""
    graded = case["how"] == "nonuniform"
    s.dz = None
    dx = s.dx
    if graded:
        m = s.shape[2] - 1 - 2 * s.ncp
        dz = [float(rng.uniform(0.2, 1.0)) * dx]
        for _ in range(m - 1):
            dz.append(min(dx, max(0.2 * dx, dz[-1] * float(rng.uniform(1 / 1.2, 1.2)))))
        s.dz = np.asarray(dz)
        full = np.concatenate([np.full(s.ncp, dz[0]), dz, np.full(s.ncp, dz[-1])])
        full = np.concatenate([full, full[-1:]])
        s.dz_full = full.astype(np.float32).astype(np.float64)
        c = 1.0 / math.sqrt(EPS_0 * MU_0)
        s.dt = float(0.99 / (c * np.sqrt(2 / dx ** 2 + 1 / float(np.min(full)) ** 2)))
    else:
        s.dt = float(dx / (C0 * np.sqrt(3.0)) * 0.99)
    s.pec_axes = "xyz" if case["how"] in ("run", "nonuniform", "decay") else ("" if s.axes == "xyz" else
                                                                              "".join(a for a in "xyz" if a not in s.axes))
    pad = [s.ncp if a in s.axes else 0 for a in "xyz"]
    # dielectric boxes in a vacuum, some of them lossy
    eps = np.ones(s.shape, np.float32)
    sig = np.zeros(s.shape, np.float32)
    lossy = case["how"] not in ("sweep",)
    for _ in range(6):
        lo, hi = [], []
        for a in range(3):
            inner = s.shape[a] - 2 * pad[a]
            n = int(rng.integers(max(2, inner // 8), max(3, inner // 3) + 1))
            lo.append(pad[a] + int(rng.integers(0, max(1, inner - n))))
            hi.append(lo[-1] + n)
        sl = tuple(slice(q, h) for q, h in zip(lo, hi))
        eps[sl] = np.float32(rng.uniform(1.0, 6.0))
        sig[sl] = np.float32(rng.uniform(0.0, 0.05) if lossy else 0.0)
    if case.get("vacuum"):
        eps[:], sig[:] = 1.0, 0.0
    s.eps, s.sig = eps, sig
    s.mu = None
    if case.get("mu"):
        s.mu = np.ones(s.shape, np.float32)
        s.mu[: s.shape[0] // 2] = np.float32(rng.uniform(1.2, 3.0))
    s.pec = None
    if case.get("sheet"):
        s.pec = np.zeros(s.shape, bool)
        k = pad[2] + max(2, (s.shape[2] - 2 * pad[2]) // 6)
        if graded:
            s.pec[:, :, k] = True
        else:
            s.pec[s.shape[0] // 4: s.shape[0] // 2, s.shape[1] // 4: s.shape[1] // 2, k:k + 2] = True

    def inner_cell():
        return tuple(int(rng.integers(p + 2, n - p - 2)) for p, n in zip(pad, s.shape))

    c = tuple(n // 2 for n in s.shape)
    comp = "ex" if graded else "ez"
    amp = float(rng.uniform(0.5, 2.0))
    wave = (_carrier(case["f0"], s.steps, s.dt, amp) if case["how"] in ("run", "nonuniform") else
            _pulse(case["f0"], s.steps, s.dt, amp, 4.0 if case["how"] == "decay" else 2.2))
    s.sources = [(c[0] - 1, c[1], c[2], comp, wave)]
    if case["how"] in ("steps", "adjoint"):
        s.sources.append((*inner_cell(), "ey", _pulse(0.6 * case["f0"], s.steps, s.dt, 0.3)))
    # probes near enough for the pulse to pass them within the pass
    reach = max(2, min(min(n - 2 * p for n, p in zip(s.shape, pad)) // 2 - 2, int(0.4 * s.steps), 14))
    s.probes = []
    for q in range(case.get("probes", 0)):
        off = [int(rng.integers(-reach, reach + 1)) for _ in range(3)]
        s.probes.append((c[0] + off[0], c[1] + off[1], c[2] + off[2], comp if q < 2 else COMPS[int(rng.integers(0, 6))]))
    s.port = (c[0] + 3, c[1], c[2]) if case.get("port") else None
    if s.port:
        s.sig[s.port] += np.float32(dx / (50.0 * dx * dx))
    nf = case.get("dft", 0)
    s.dft = [(2, c[2] + 1, comp, np.linspace(0.5 * case["f0"], 1.5 * case["f0"], nf).astype(np.float32))] if nf else []
    s.box = None
    if case.get("box"):
        b = case["box"]
        bx, by = min(b, s.shape[0] - 2 * pad[0] - 4), min(b, s.shape[1] - 2 * pad[1] - 4)
        i0, j0, k0 = (s.shape[0] - bx) // 2, (s.shape[1] - by) // 2, c[2]
        s.box = (i0, i0 + bx, j0, j0 + by, k0, k0 + 2)
        s.eps[i0:i0 + bx, j0:j0 + by, k0:k0 + 2] = (1.0 + 3.4 * rng.random((bx, by, 2))).astype(np.float32)
    s.freqs = np.array([0.8, 1.0, 1.2]) * case["f0"]
    s.init_seed = int(rng.integers(1 << 30)) if case["how"] == "steps" else None
    return s


def _start_fields(s, dtype):
    """Fields of a march under way: a few standing waves per component, E of order one and H of E / 377."""
    rng = np.random.default_rng([s.init_seed, 11])
    dev = torch.device("cuda")
    out = []
    for c in range(6):
        f = torch.zeros(s.shape, device=dev, dtype=torch.float32)
        for _ in range(3):
            w = []
            for n in s.shape:
                k, p = 2 * math.pi / rng.uniform(9.0, 45.0), rng.uniform(0, 2 * math.pi)
                w.append(torch.from_numpy(np.cos(k * np.arange(n) + p).astype(np.float32)).to(dev))
            a = float(rng.uniform(0.2, 0.6)) / (1.0 if c < 3 else 377.0)
            f += (a * w[0])[:, None, None] * w[1][None, :, None] * w[2][None, None, :]
        out.append(f.to(dtype))
    return out


def _ntff_box(case):
    n, p = (case["nx"], case["ny"], case["nz"]), case["ncp"] + 3
    return (p, p, p), tuple(v - p for v in n)


def _angles():
    return np.linspace(0.05, math.pi - 0.05, 25), np.linspace(0.0, 2 * math.pi, 36, endpoint=False)


def _ntff_freqs(case):
    return np.linspace(0.8 * case["f0"], 1.2 * case["f0"], case["ntff"]).astype(np.float32)


def _flux_region(case):
    p = case["ncp"]
    f = np.linspace(0.7 * case["f0"], 1.3 * case["f0"], case["flux"])
    return case["nx"] // 2 + 4, p, case["ny"] - p, p, case["nz"] - p, f


def _sweep_sizes(case):
    r = np.random.default_rng([case["n_inst"], case["n_lo"], case["n_hi"]])
    return [int(n) + 17 for n in r.integers(case["n_lo"], case["n_hi"] + 1, case["n_inst"])]


def _sweep_scenes(case, seed):
    out = []
    for q, n in enumerate(_sweep_sizes(case)):
        s = _scene(dict(case, nx=n, ny=n, nz=n, box=16, probes=0), int(seed) * 64 + q)
        c = n // 2
        i0, i1, j0, j1, _, _ = s.box
        s.box = (c - 4, c + 4, j0, j1, c, c + 2)
        # source and probes on either side of the region, within reach of the pass
        s.sources = [(c - 6, c, c, "ez", _pulse(case["f0"] * 4, s.steps, s.dt, 1.0))]
        s.probes = [(c + 6, c + d, c, "ez") for d in (-4, -1, 1, 4)]
        out.append(s)
    return out


# ---------------------------------------------------------------------------
# prepare and run


def _grid(s):
    if s.dz is not None:
        m = [(n - 1 - 2 * s.ncp) * s.dx for n in s.shape[:2]]
        g = rfx_b200.make_nonuniform_grid(tuple(m), s.dz, s.dx, cpml_layers=s.ncp)
    else:
        dom = tuple((n - 1 - (2 * s.ncp if a in s.axes else 0) - 0.5) * s.dx for a, n in zip("xyz", s.shape))
        g = rfx_b200.Grid(freq_max=20e9, domain=dom, dx=s.dx, cpml_layers=s.ncp, cpml_axes=s.axes or "xyz")
    assert tuple(g.shape) == s.shape, (g.shape, s.shape)
    return g


def _materials(s):
    mu = s.mu if s.mu is not None else np.ones(s.shape, np.float32)
    return rfx_b200.MaterialArrays(s.eps, s.sig, mu)


def prepare(case, seed):
    st = _Scene()
    st.case = case
    if case["how"] == "sweep":
        scenes = _sweep_scenes(case, seed)
        insts = [SweepInstance(grid=_grid(s), eps_r=s.eps, sigma=s.sig, sources=s.sources, probes=s.probes, box=s.box,
                               freqs=s.freqs) for s in scenes]
        st.sweep = Sweep(insts, case["steps"])
        return st
    s = st.scene = _scene(case, seed)
    g = st.grid = _grid(s)
    mats = st.mats = _materials(s)
    planes = [rfx_b200.init_dft_plane_probe(a, ix, c, f, g.shape) for (a, ix, c, f) in s.dft]
    how = case["how"]
    if how in ("run", "decay"):
        kw = st.kw = dict(boundary="cpml" if s.ncp else "pec", sources=[rfx_b200.SourceSpec(*q) for q in s.sources],
                          probes=[rfx_b200.ProbeSpec(*p) for p in s.probes], dft_planes=planes or None,
                          pec_mask=s.pec)
        if how == "decay":
            return st
        kw["return_state"] = bool(case.get("state"))
        if s.port:
            kw["lumped_port_sparams"] = [rfx_b200.LumpedPortSParamSpec(*s.port, "ez", s.freqs, 50.0)]
        if case.get("ntff"):
            lo, hi = _ntff_box(case)
            kw["ntff"] = rfx_b200.NTFFBox.from_grid(g, i_lo=lo[0], i_hi=hi[0], j_lo=lo[1], j_hi=hi[1], k_lo=lo[2],
                                                    k_hi=hi[2], freqs=_ntff_freqs(case))
        if case.get("flux"):
            ix, l1, h1, l2, h2, f = _flux_region(case)
            kw["flux_monitors"] = [rfx_b200.init_flux_monitor(0, ix, f, g.shape, s.dx, s.dx, lo1=l1, hi1=h1, lo2=l2,
                                                              hi2=h2)]
    elif how == "nonuniform":
        st.kw = dict(sources=s.sources, probes=s.probes, dft_planes=planes or None, pec_mask=s.pec)
    elif how == "steps":
        st.dev = prepare_device_run(g, mats, s.steps, cpml_axes=s.axes, pec_axes=s.pec_axes, sources=s.sources,
                                    probes=s.probes, dft_planes=planes, pec_mask=s.pec, dft_time_offset=1)
        st.fields = _start_fields(s, torch.float32)
    else:
        st.runner = AdjointRunner(g, mats, s.steps, sources=s.sources, probes=s.probes, box=s.box, pec_axes="",
                                  dft_planes=planes, checkpoint_every=case["every"] or None)
        i0, i1, j0, j1, k0, k1 = s.box
        st.eps = torch.from_numpy(s.eps[i0:i1, j0:j1, k0:k1].copy()).cuda().requires_grad_(True)
        tab = np.stack([q[4] for q in s.sources], axis=-1)
        st.src = torch.from_numpy(np.ascontiguousarray(tab)).cuda().requires_grad_(True)
        # the cotangents of a linear objective (weights of the probe samples and of the DFT plane)
        rng = np.random.default_rng([int(seed), 13])
        st.g_ts = torch.from_numpy(rng.standard_normal((s.steps, len(s.probes))).astype(np.float32)).cuda()
        st.g_dft = [torch.from_numpy(_complex(rng, p.accumulator.shape)).cuda() for p in planes]
    return st


def _complex(rng, shape):
    return (1e9 * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape))).astype(np.complex64)


def run(st):
    case = st.case
    how = case["how"]
    if how == "sweep":
        Js, grads = st.sweep.run()
        return {"objective": Js, "grad": grads}
    if how == "run":
        r = rfx_b200.run(st.grid, st.mats, case["steps"], **st.kw)
        out = {"trace": r.time_series}
        if r.state is not None:
            out["state"] = [getattr(r.state, c) for c in COMPS]
        if r.dft_planes:
            out["dft"] = [p.accumulator for p in r.dft_planes]
        if r.lumped_port_sparams:
            out["port"] = list(r.lumped_port_sparams[0][1])
        if r.flux_monitors:
            m = r.flux_monitors[0]
            out["flux"] = [m.e1_dft, m.e2_dft, m.h1_dft, m.h2_dft]
        if r.ntff_data is not None:
            out["ntff"] = list(r.ntff_data[:6])
            ff = rfx_b200.compute_far_field(r.ntff_data, st.kw["ntff"], st.grid, *_angles())
            out["far"] = [ff.E_theta, ff.E_phi]
        return out
    if how == "decay":
        r = rfx_b200.run_until_decay(st.grid, st.mats, decay_by=1e-2, check_interval=50, min_steps=100,
                                     max_steps=case["steps"], **st.kw)
        # the length depends on the scene: zeros up to the cap
        trace = np.pad(r.time_series, ((0, case["steps"] - len(r.time_series)), (0, 0)))
        return {"trace": trace, "state": [getattr(r.state, c) for c in COMPS], "steps": int(r.state.step)}
    if how == "nonuniform":
        r = rfx_b200.run_nonuniform(st.grid, st.mats, case["steps"], **st.kw)
        out = {"trace": r["time_series"], "state": [getattr(r["state"], c) for c in COMPS]}
        if "dft_planes" in r:
            out["dft"] = [p.accumulator for p in r["dft_planes"]]
        return out
    if how == "steps":
        d = st.dev
        d.plan.reset()
        d.plan.load_fields(st.fields)
        for a in d.dft_accs:
            a.zero_()
        d.plan.advance(0, case["steps"], d.src_table, d.probe_out, d.dft_accs, d.dft_phases)
        return {"trace": d.probe_out, "state": d.plan.store_fields(), "dft": list(d.dft_accs)}
    r = st.runner
    if case["every"]:   # the explicit pair of passes
        r.set_box_eps(st.eps.detach())
        ts = r.forward(st.src.detach())
        grad, src = r.backward(st.g_ts, g_dft=st.g_dft or None)
        return {"trace": ts, "dft": list(r.dft_accs), "grad": grad, "src_grad": src}
    outs = FDTDFunction.apply(st.eps, st.src, r)   # torch.autograd
    outs = outs if isinstance(outs, tuple) else (outs,)
    grad, src = torch.autograd.grad(outs, (st.eps, st.src), [st.g_ts, *st.g_dft])
    return {"trace": outs[0].detach(), "dft": [o.detach() for o in outs[1:]], "grad": grad, "src_grad": src}


# ---------------------------------------------------------------------------
# the same march in float64


class _March:
    """The Yee / CPML march of a scene in float64 torch, differentiable in eps and the source table."""

    def __init__(self, s):
        self.s = s
        dev = self.dev = torch.device("cuda")
        f8 = dict(device=dev, dtype=torch.float64)
        nx, ny, nz = s.shape
        inv = float(np.float32(1.0) / np.float32(s.dx))
        xe = xh = torch.full((nx, 1, 1), inv, **f8)
        ye = yh = torch.full((1, ny, 1), inv, **f8)
        ze = zh = torch.full((1, 1, nz), inv, **f8)
        cells = [s.dx, s.dx, s.dx, s.dx, s.dx, s.dx]
        if s.dz is not None:
            d = s.dz_full
            h = np.concatenate([1.0 / d[:-1], [0.0]])
            e = np.concatenate([1.0 / d[:1], 2.0 / (d[:-1] + d[1:])])
            zh, ze = torch.from_numpy(h).to(dev)[None, None], torch.from_numpy(e).to(dev)[None, None]
            cells[4:] = [float(d[0]), float(d[-1])]
            for n, a in ((nx, 0), (ny, 1)):
                t = np.full(n, inv)
                t[-1] = 0.0
                t = torch.from_numpy(t).to(dev)
                if a == 0:
                    xh = t[:, None, None]
                else:
                    yh = t[None, :, None]
        self.inv_e, self.inv_h = (xe, ye, ze), (xh, yh, zh)
        self.ch = s.dt / (MU_0 if s.mu is None else MU_0 * torch.from_numpy(s.mu).to(**f8))
        self.sig = torch.from_numpy(s.sig).to(**f8)
        self.slabs = []          # (axis, face index range, b, c / cell) of every absorbing face
        n = s.ncp
        for a, ax in enumerate("xyz"):
            if ax not in s.axes:
                continue
            for side in range(2):
                cell = cells[2 * a + side]
                rho = 1.0 - np.arange(n) / max(n - 1, 1)
                smax = -math.log(1e-15) * 4 / (2.0 * math.sqrt(MU_0 / EPS_0) * n * cell)
                sg, al = smax * rho ** 3, 0.05 * (1.0 - rho)
                b = np.exp(-(sg + al) * s.dt / EPS_0)
                c = np.where(sg + al > 1e-30, sg * (b - 1.0) / np.maximum(sg + al, 1e-300), 0.0) / cell
                if side:
                    b, c = b[::-1].copy(), c[::-1].copy()
                shp = [1, 1, 1]
                shp[a] = n
                self.slabs.append((a, 0 if side == 0 else s.shape[a] - n,
                                   torch.from_numpy(b).to(dev).view(shp), torch.from_numpy(c).to(dev).view(shp)))
        self.mask = None
        if s.pec is not None:
            m = torch.from_numpy(s.pec).to(dev)
            self.mask = []
            for a in range(3):
                nb = torch.zeros_like(m)
                k = s.shape[a]
                nb.narrow(a, 1, k - 1).logical_or_(m.narrow(a, 0, k - 1))
                nb.narrow(a, 0, k - 1).logical_or_(m.narrow(a, 1, k - 1))
                self.mask.append((~(m & nb)).to(torch.float64))

    def coefficients(self, eps):
        s = self.s
        e = eps * EPS_0
        q = self.sig * s.dt / (2.0 * e)
        return (1 - q) / (1 + q), (s.dt / e) / (1 + q), s.dt / e

    def zero(self, fields=None):
        z = fields or [torch.zeros(self.s.shape, device=self.dev, dtype=torch.float64) for _ in range(6)]
        psi = []
        for a, _, _, _ in self.slabs:
            shp = list(self.s.shape)
            shp[a] = self.s.ncp
            psi += [torch.zeros(shp, device=self.dev, dtype=torch.float64) for _ in range(4)]
        return list(z), psi

    @staticmethod
    def _diff(f, a, back):
        shp = list(f.shape)
        shp[a] = 1
        z = torch.zeros(shp, device=f.device, dtype=f.dtype)
        return torch.diff(f, dim=a, prepend=z) if back else torch.diff(f, dim=a, append=z)

    # (component, sign) that the correction of the derivative of component t along axis a goes into, per side
    H_TERMS = {0: ((2, 1, +1), (1, 2, -1)), 1: ((2, 0, -1), (0, 2, +1)), 2: ((1, 0, +1), (0, 1, -1))}
    E_TERMS = {0: ((2, 1, -1), (1, 2, +1)), 1: ((2, 0, +1), (0, 2, -1)), 2: ((1, 0, -1), (0, 1, +1))}

    def _half(self, src, dst, scale, decay, inv, back, psi, o, cpml_scale, terms, sign):
        """dst <- decay * dst + sign * scale * curl src, then the CPML corrections scaled by cpml_scale."""
        d = {}
        for a in range(3):
            for t in range(3):
                if t != a:
                    d[a, t] = self._diff(src[t], a, back)
        new = []
        for q, (a1, t1, a2, t2) in enumerate(((1, 2, 2, 1), (2, 0, 0, 2), (0, 1, 1, 0))):
            curl = d[a1, t1] * inv[a1] - d[a2, t2] * inv[a2]
            base = dst[q] if decay is None else decay * dst[q]
            new.append(base + sign * scale * curl)
        out_psi = []
        for f, (a, lo, b, c) in enumerate(self.slabs):
            n = self.s.ncp
            for q, (t, into, sg) in enumerate(terms[a]):
                p = b * psi[4 * f + o + q] + c * d[a, t].narrow(a, lo, n)
                out_psi.append(p)
                k = cpml_scale if not torch.is_tensor(cpml_scale) else cpml_scale.narrow(a, lo, n)
                new[into].narrow(a, lo, n).add_(sg * k * p)
        return new, out_psi

    def step(self, F, psi, coef, n, src):
        s = self.s
        ca, cb, ce = coef
        H, pH = self._half(F[:3], F[3:], self.ch, None, self.inv_h, False, psi, 0, self.ch, self.H_TERMS, -1.0)
        E, pE = self._half(H, F[:3], cb, ca, self.inv_e, True, psi, 2, ce, self.E_TERMS, +1.0)
        psi = []
        for f in range(len(self.slabs)):
            psi += [pH[2 * f], pH[2 * f + 1], pE[2 * f], pE[2 * f + 1]]
        for a in range(3):
            if "xyz"[a] in s.pec_axes:
                for t in range(3):
                    if t != a:
                        for at in (0, s.shape[a] - 1):
                            E[t].select(a, at).zero_()
        if "z" in s.pec_axes:
            E[2].select(2, s.shape[2] - 1).zero_()
        if self.mask is not None:
            E = [e * m for e, m in zip(E, self.mask)]
        pre = None
        if s.port is not None:
            i, j, k = s.port
            pre = torch.stack([-E[2][i, j, k], H[1][i, j, k] - H[1][i - 1, j, k] - H[0][i, j, k] + H[0][i, j - 1, k]])
        for q, (i, j, k, c, _) in enumerate(s.sources):
            E[COMPS.index(c)][i, j, k] += src[n, q]
        return E + H, psi, pre

    def source_table(self):
        return torch.from_numpy(np.stack([q[4] for q in self.s.sources], -1)).to(self.dev, torch.float64)

    def sample(self, F):
        if not self.s.probes:
            return torch.zeros(0, device=self.dev, dtype=torch.float64)
        return torch.stack([F[COMPS.index(c)][i, j, k] for (i, j, k, c) in self.s.probes])

    def plane(self, F, q, n, offset):
        a, ix, c, fr = self.s.dft[q]
        ph = -2.0 * math.pi * fr.astype(np.float64) * (n + offset) * self.s.dt
        w = torch.from_numpy(np.exp(1j * ph) * self.s.dt).to(self.dev)
        return w[:, None, None] * F[COMPS.index(c)].select(a, ix)[None]


def exact(case, seed):
    if case["how"] == "sweep":
        Js, gs = [], []
        for s in _sweep_scenes(case, seed):
            m = _March(s)

            def objective(ts, s=s):
                n = torch.arange(s.steps, device=ts.device, dtype=torch.float64)
                f = torch.from_numpy(s.freqs).to(ts.device)
                ph = torch.exp(-2j * math.pi * f[:, None] * n[None, :] * s.dt) * s.dt
                X = ph @ ts.to(torch.complex128)
                return (X.real ** 2 + X.imag ** 2).sum()
            J, g, _, _, _ = _gradients(m, objective, None, 10)
            Js.append(J)
            gs.append(g)
        return {"objective": Js, "grad": gs}
    s = _scene(case, seed)
    m = _March(s)
    offset = 0 if case["how"] == "nonuniform" else 1
    if case["how"] == "adjoint":
        rng = np.random.default_rng([int(seed), 13])
        g_ts = torch.from_numpy(rng.standard_normal((s.steps, len(s.probes))).astype(np.float32)).to(m.dev).double()
        g_dft = [torch.from_numpy(_complex(rng, (len(fr), s.shape[0], s.shape[1]))).to(m.dev).to(torch.complex128)
                 for (_, _, _, fr) in s.dft]
        _, grad, src, ts, accs = _gradients(m, lambda t: (t * g_ts).sum(), g_dft, 10)
        return {"trace": ts, "dft": accs, "grad": grad, "src_grad": src}
    with torch.no_grad():
        F, psi = m.zero(_start_fields(s, torch.float64) if case["how"] == "steps" else None)
        coef = m.coefficients(torch.from_numpy(s.eps).to(m.dev).double())
        src = m.source_table()
        accs = [0.0 for _ in s.dft]
        rows, ports = [], []
        obs = _Observers(case, s, m) if (case.get("ntff") or case.get("flux")) else None
        peak, below = 0.0, 0
        p = s.ncp
        done = s.steps
        for n in range(s.steps):
            F, psi, pre = m.step(F, psi, coef, n, src)
            rows.append(m.sample(F))
            if pre is not None:
                ports.append(pre)
            accs = [a + m.plane(F, q, n, offset) for q, a in enumerate(accs)]
            if obs:
                obs.add(F, n)
            if case["how"] == "decay" and n % 50 == 0 and n >= 99:
                u = float(sum(f[p:-p, p:-p, p:-p].square().sum() for f in F))
                peak = max(peak, u)
                below = below + 1 if u < 1e-2 * peak else 0
                if below >= 2:
                    done = n + 1
                    break
        out = {"trace": torch.nn.functional.pad(torch.stack(rows), (0, 0, 0, s.steps - len(rows)))}
        if case["how"] in ("decay", "nonuniform", "steps") or case.get("state"):
            out["state"] = F
        if case["how"] == "decay":
            out["steps"] = done
        if accs or case["how"] == "steps":
            out["dft"] = accs
        if ports:
            v = torch.stack(ports).cpu().numpy() * s.dx
            ph = np.exp(-2j * math.pi * s.freqs[:, None] * (np.arange(s.steps)[None] * s.dt)) * s.dt
            out["port"] = [ph @ v[:, 0], ph @ v[:, 1]]
        if obs:
            out.update(obs.result())
        return out


def _gradients(m, objective, g_dft, chunk):
    """(objective, d/d eps over the box, d/d source table, traces, DFT planes) by autograd, recomputing chunks."""
    from torch.utils.checkpoint import checkpoint
    s = m.s
    i0, i1, j0, j1, k0, k1 = s.box
    base = torch.from_numpy(s.eps).to(m.dev).double()
    eps_box = base[i0:i1, j0:j1, k0:k1].clone().requires_grad_(True)
    src = m.source_table().requires_grad_(True)
    np_ = len(m.slabs) * 4

    def part(n0, n1, eps_box, src, *state):
        eps = base.clone()
        eps[i0:i1, j0:j1, k0:k1] = eps_box
        coef = m.coefficients(eps)
        F, psi, accs = list(state[:6]), list(state[6:6 + np_]), list(state[6 + np_:])
        rows = []
        for n in range(n0, n1):
            F, psi, _ = m.step(F, psi, coef, n, src)
            rows.append(m.sample(F))
            accs = [a + m.plane(F, q, n, 1) for q, a in enumerate(accs)]
        return (torch.stack(rows), *F, *psi, *accs)

    F, psi = m.zero()
    accs = [torch.zeros((len(fr), s.shape[0], s.shape[1]), device=m.dev, dtype=torch.complex128) for (_, _, _, fr) in s.dft]
    state, rows = [*F, *psi, *accs], []
    for n0 in range(0, s.steps, chunk):
        r = checkpoint(part, n0, min(s.steps, n0 + chunk), eps_box, src, *state, use_reentrant=False)
        rows.append(r[0])
        state = list(r[1:])
    ts = torch.cat(rows)
    accs = state[6 + np_:]
    J = objective(ts)
    total = J
    for a, g in zip(accs, g_dft or []):
        total = total + (a.real * g.real + a.imag * g.imag).sum()
    ge, gs = torch.autograd.grad(total, (eps_box, src))
    return J.detach(), ge, gs, ts.detach(), [a.detach() for a in accs]


class _Observers:
    """NTFF faces, a flux monitor on an x plane, and the far field of the faces, in float64."""

    def __init__(self, case, s, m):
        self.case, self.s, self.m = case, s, m
        self.faces = [0.0] * 6
        self.flux = 0.0

    def add(self, F, n):
        s, dev, dt = self.s, self.m.dev, self.s.dt
        if self.case.get("ntff"):
            lo, hi = _ntff_box(self.case)
            f = _ntff_freqs(self.case).astype(np.float64)
            we = torch.from_numpy(np.exp(-2j * math.pi * f * n * dt) * dt).to(dev)
            wh = torch.from_numpy(np.exp(-2j * math.pi * f * (n + 0.5) * dt) * dt).to(dev)
            for q in range(6):
                a = q // 2
                t = [x for x in range(3) if x != a]
                at = hi[a] if q % 2 else lo[a]
                v = [F[c].select(a, at)[lo[t[0]]:hi[t[0]], lo[t[1]]:hi[t[1]]] for c in (t[0], t[1], 3 + t[0], 3 + t[1])]
                v = torch.stack(v, -1)
                w = torch.stack([we, we, wh, wh], -1)
                self.faces[q] = self.faces[q] + w[:, None, None, :] * v[None]
        if self.case.get("flux"):
            ix, l1, h1, l2, h2, f = _flux_region(self.case)
            t = (n + 1) * dt
            we = torch.from_numpy(np.exp(-2j * math.pi * f * t) * dt).to(dev)
            wh = torch.from_numpy(np.exp(-2j * math.pi * f * (t - 0.5 * dt)) * dt).to(dev)
            e = torch.stack([F[c][ix, l1:h1, l2:h2] for c in (1, 2)])
            h = torch.stack([0.5 * (F[c][ix - 1, l1:h1, l2:h2] + F[c][ix, l1:h1, l2:h2]) for c in (4, 5)])
            self.flux = self.flux + torch.cat([we[None, :, None, None] * e[:, None], wh[None, :, None, None] * h[:, None]])

    def result(self):
        out = {}
        if self.case.get("flux"):
            out["flux"] = list(self.flux)
        if not self.case.get("ntff"):
            return out
        s, dev = self.s, self.m.dev
        lo, hi = _ntff_box(self.case)
        f = _ntff_freqs(self.case).astype(np.float64)
        th, ph = (torch.from_numpy(a).to(dev) for a in _angles())
        TH, PH = torch.meshgrid(th, ph, indexing="ij")
        sth, cth, sph, cph = TH.sin(), TH.cos(), PH.sin(), PH.cos()
        r = torch.stack([sth * cph, sth * sph, cth], -1).reshape(-1, 3)
        N = L = 0.0
        for q in range(6):
            a, sg = q // 2, (1.0 if q % 2 else -1.0)
            t = [x for x in range(3) if x != a]
            X = self.faces[q].reshape(len(f), -1, 4)
            full = torch.zeros((2, len(f), X.shape[1], 3), device=dev, dtype=torch.complex128)
            for w in range(2):
                full[w][..., t[0]], full[w][..., t[1]] = X[..., 2 * w], X[..., 2 * w + 1]
            nrm = torch.zeros(3, device=dev, dtype=torch.complex128)
            nrm[a] = sg
            J = torch.linalg.cross(nrm.expand_as(full[1]), full[1]) * s.dx ** 2
            M = -torch.linalg.cross(nrm.expand_as(full[0]), full[0]) * s.dx ** 2
            g = [torch.arange(lo[x], hi[x], device=dev, dtype=torch.float64) for x in t]
            G = torch.meshgrid(*g, indexing="ij")
            pos = [None] * 3
            pos[t[0]], pos[t[1]] = G[0], G[1]
            pos[a] = torch.full_like(G[0], float(hi[a] if q % 2 else lo[a]))
            pos = (torch.stack(pos, -1).reshape(-1, 3) - s.ncp) * s.dx
            dot = r @ pos.T
            parts = [torch.polar(torch.ones_like(dot), 2 * math.pi * float(v) / C0 * dot) for v in f]
            N = N + torch.stack([p @ J[i] for i, p in enumerate(parts)])
            L = L + torch.stack([p @ M[i] for i, p in enumerate(parts)])
        eta = math.sqrt(MU_0 / EPS_0)
        tv = torch.stack([cth * cph, cth * sph, -sth], -1).reshape(-1, 3)
        pv = torch.stack([-sph, cph, torch.zeros_like(sth)], -1).reshape(-1, 3)
        jk = torch.from_numpy(2j * math.pi * f / C0).to(dev)[:, None]
        dot3 = lambda A, v: (A * v).sum(-1)   # noqa: E731
        Et = -jk / (4 * math.pi) * (dot3(L, pv) + eta * dot3(N, tv))
        Ep = jk / (4 * math.pi) * (dot3(L, tv) - eta * dot3(N, pv))
        shp = (len(f), len(th), len(ph))
        out["ntff"] = [x for x in self.faces]
        out["far"] = [Et.reshape(shp), Ep.reshape(shp)]
        return out
