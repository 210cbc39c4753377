"""The work that a user of this framework has it do, as cases that can be timed and compared.

Four kinds of call, each through the public entry point a program uses:

* ``batch``   ``Engine.run_batch`` / ``run_batch_ions`` / ``sweep.run_sweep``: scan points in, outcomes
              (or final ion states) out, on the mixed-precision and on the FP64 engine;
* ``states``  ``Engine.run_ions``: the caller's ion states advanced by a number of steps;
* ``tandem``  ``TandemModel.advance``: a pulse of tracks through splitter, nine channels and combiner;
* ``solve``   ``Fields.build`` on the device: the field bases of a geometry from its electrodes.

A program solves a geometry once and keeps an engine on it; so ``prepare`` solves each geometry once
per process, and makes an engine, jobs and launch states of its own for every state.
"""
import math

import numpy as np
import torch

import multiq_workbench_gb300 as mq

AMU, QE = 1.6605390666e-27, 1.602176634e-19
FIG4_DC = [0.0, 5.0, -5.0, 0.0]
S14_DC = [18.0, 24.0, 15.0, 20.0]
# Outcome columns that are counts, and those that are means over a job's ions.
COUNTS = ("n", "crashed", "returned", "transmitted", "left", "timeout")
MEANS = ("mean_coll", "mean_time")
# Mean steps an ion of each physics makes before it ends (to its step cap), for the estimate of work.
MEAN_STEPS = {"corrected": 270, "half_kick": 640, "legacy": 13600, "s14": 18000, "s14_point": 5700}


def listed():
    return [
        # One operating point, 1,000 ions of m/z 499 to completion: the smallest thing a user runs.
        {"name": "point", "kind": "batch", "physics": "half_kick", "engine": "mixed", "h": 0.1, "jobs": 1, "ions": 1000, "want": "counts"},
        # The mass scan with the corrected update: ions end within few RF periods, so launches, copies
        # and set-up show. Per-ion final states come back, as for a class-by-class comparison.
        {"name": "mass_scan_corrected", "kind": "batch", "physics": "corrected", "engine": "mixed", "h": 0.1, "jobs": 25, "ions": 1000, "want": "ions"},
        # The legacy Fig. 4 mass scan: 26 m/z x 1,000 ions, every legacy switch, 20,000-step cap.
        {"name": "legacy_fig4_scan", "kind": "batch", "physics": "legacy", "engine": "mixed", "h": 0.1, "jobs": 26, "ions": 1000, "want": "counts"},
        # A resonance sweep at the S14 point: 31 tones x 2 species, 2,000 ions a tone, 75,000-step cap.
        {"name": "s14_resonance_sweep", "kind": "batch", "physics": "s14", "engine": "mixed", "h": 0.1, "jobs": 31, "ions": 2000, "want": "sweep"},
        # The production sweep: 64 tones x 8 amplitudes x 32 m/z x 256 ions, 4.2 million ions in one call.
        {"name": "batched_sweep", "kind": "batch", "physics": "half_kick", "engine": "mixed", "h": 0.1, "jobs": 16384, "ions": 256, "want": "counts"},
        # The grid-resolution study's middle grid: 1,024 seeds x 1,000 ions on 49.6 million nodes.
        {"name": "fine_grid_study", "kind": "batch", "physics": "half_kick", "engine": "mixed", "h": 0.05, "jobs": 1024, "ions": 1000, "want": "counts"},
        # The mass scan on the FP64 engine: the reference results that mixed runs are checked against.
        {"name": "mass_scan_fp64", "kind": "batch", "physics": "half_kick", "engine": "f64", "h": 0.1, "jobs": 25, "ions": 1000, "want": "ions"},
        # The S14 validation point on the FP64 engine, a few thousand ions at one setting.
        {"name": "s14_point_fp64", "kind": "batch", "physics": "s14_point", "engine": "f64", "h": 0.1, "jobs": 1, "ions": 20000, "want": "counts"},
        # A caller that keeps the ion states itself and moves them on by 500 steps at a time, no gas.
        {"name": "advance_states", "kind": "states", "engine": "mixed", "ions": 65537, "steps": 500},
        # The tandem as the interactive program has it: 180 tracks, FP64, a hundred steps a frame or so.
        {"name": "tandem_live", "kind": "tandem", "engine": "f64", "tracks": 180, "steps": 100, "fine": False},
        # A pulse through the tandem on the mixed engine.
        {"name": "tandem_pulse", "kind": "tandem", "engine": "mixed", "tracks": 262144, "steps": 1000, "fine": True},
        # RF and AC bases of a channel whose rods are slightly out of place, at the usual spacing.
        {"name": "field_solve", "kind": "solve", "h": 0.1, "bases": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("batch", "batch", "batch", "batch64", "states", "tandem", "solve"))
    if kind == "batch":
        physics = rng.choice(("corrected", "half_kick", "legacy", "s14"))
        most = {"corrected": 2000000, "half_kick": 4000000, "legacy": 200000, "s14": 200000}[physics]
        n = _log(rng, 200, most)
        if physics == "s14":
            jobs = rng.choice((7, 16, 31, 61))
            return {"kind": "batch", "physics": physics, "engine": "mixed", "h": 0.1, "jobs": jobs, "ions": max(2, n // jobs), "want": "sweep"}
        jobs = min(_log(rng, 1, 4096), max(1, n // 16))
        h = rng.choice((0.1, 0.1, 0.16, 0.05)) if physics == "half_kick" else 0.1
        want = "ions" if n <= 300000 and rng.random() < 0.4 else "counts"
        return {"kind": "batch", "physics": physics, "engine": "mixed", "h": h, "jobs": jobs, "ions": max(1, n // jobs), "want": want}
    if kind == "batch64":
        physics = rng.choice(("corrected", "half_kick", "legacy", "s14_point"))
        n = _log(rng, 100, {"corrected": 100000, "half_kick": 60000, "legacy": 6000, "s14_point": 12000}[physics])
        jobs = 1 if physics == "s14_point" else min(_log(rng, 1, 64), n)
        return {"kind": "batch", "physics": physics, "engine": "f64", "h": 0.1, "jobs": jobs, "ions": max(1, n // jobs), "want": rng.choice(("ions", "counts"))}
    if kind == "states":
        engine = rng.choice(("mixed", "mixed", "f64"))
        return {"kind": "states", "engine": engine, "ions": _log(rng, 33, 500000 if engine == "mixed" else 60000), "steps": _log(rng, 17, 1500 if engine == "mixed" else 600)}
    if kind == "tandem":
        engine = rng.choice(("mixed", "f64"))
        tracks = _log(rng, 50, 400000 if engine == "mixed" else 20000)
        return {"kind": "tandem", "engine": engine, "tracks": tracks, "steps": _log(rng, 20, 1000 if engine == "mixed" else 500), "fine": False}
    return {"kind": "solve", "h": rng.choice((0.08, 0.1, 0.125, 0.16, 0.2, 0.25, 0.32)), "bases": rng.choice((2, 3, 4))}


# ---------------------------------------------------------------- what a program keeps

_FIELDS = {}   # solved geometries of this process, by name and spacing


def _fields(name, h):
    key = (name, h)
    if key not in _FIELDS:
        nxy = int(round(16.0 / h))
        geom = mq.Geom.s14("code", hole_d=7.0, h_mm=h, n_xy=nxy) if name == "s14" else mq.Geom.with_spacing(h)
        _FIELDS[key] = mq.Fields.build(geom, bases=None if name == "s14" else [0, 1, 3, 4], cache=False, device=0)
    return _FIELDS[key]


def _precision(case):
    return mq.PREC_F64 if case["engine"] == "f64" else mq.PREC_MIXED


def _physics(name):
    if name == "legacy":
        ph = mq.Physics.legacy(0.133322)
        ph.t_max = 20000 * ph.dt
        return ph
    if name == "s14_point":
        ph = mq.Physics.correct(0.1)
        ph.t_max = 3e-3
        return ph
    return mq.Physics(legacy_force=name == "half_kick", pressure_pa=0.133322, temp_k=300.0, dt=1e-7, t_max=20000 * 1e-7,
                      launch=mq.LAUNCH_GAUSSIAN, sigma_mm=0.1, z_inject_mm=1.0)


def _scan_jobs(physics, njobs, ions, seed):
    """The scan points of a batch: m/z over the Fig. 4 range, and, where there are many points, tones and amplitudes too."""
    base = 1000003 * int(seed)
    jobs = []
    if physics == "s14_point":
        sp, drive = mq.Species(2.0 * 863.473, 2.0, 425.0), mq.RfAc(70.0, 500e3, 0.35, 84.25e3)
        return [mq.Job(sp, drive, ions, base + k) for k in range(njobs)]
    if physics == "legacy":
        for k in range(njobs):
            mz = 475.0 + 2.0 * (k % 26)
            jobs.append(mq.Job(mq.Species(mz * 5.0, 5.0, 0.0), mq.RfAc(100.0, 500e3, 0.5, 100e3), ions, base + 1000 * (k // 26) + int(mz)))
        return jobs
    nm = min(32, njobs)
    nv = min(8, max(1, njobs // nm))
    nf = max(1, njobs // (nm * nv))
    sweep = njobs > 2048   # the production sweep; smaller scans have one drive
    for k in range(njobs):
        m, v, f = k % nm, (k // nm) % nv, (k // (nm * nv)) % nf
        mz = 499.0 if njobs == 1 else (470.0 if sweep else 475.0) + 2.0 * m
        drive = (mq.RfAc(100.0, 500e3, 0.1 + 0.9 * v / max(1, nv - 1), 80e3 + 40e3 * f / max(1, nf - 1)) if sweep
                 else mq.RfAc(100.0, 500e3, 0.5, 100e3))
        jobs.append(mq.Job(mq.Species(mz, 1.0, 2.95 * mz ** (2.0 / 3.0)), drive, ions, base + k))
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        s14 = case["physics"] in ("s14", "s14_point")
        fields = _fields("s14" if s14 else "fig4", case["h"])
        eng = mq.Engine(fields, _precision(case))
        if case["want"] == "sweep":
            preset = mq.sweep.SweepPreset.s14()
            n = case["jobs"]
            cfg = mq.sweep.SweepCfg(70.0, 100.0, 30.0 / (n - 1), ions_per_point=case["ions"])
            return {"case": case, "eng": eng, "preset": preset, "cfg": cfg, "ph": mq.sweep.sweep_physics(preset.pressure_pa), "seed": 1000003 * int(seed)}
        jobs = mq.JobTable.from_jobs(_scan_jobs(case["physics"], case["jobs"], case["ions"], seed))
        return {"case": case, "eng": eng, "jobs": jobs, "dc": S14_DC if s14 else FIG4_DC, "ph": _physics(case["physics"])}
    if kind == "states":
        fields = _fields("fig4", 0.1)
        eng = mq.Engine(fields, _precision(case))
        eng.set_dc(FIG4_DC)
        ph = _physics("half_kick")
        ph.pressure_pa = 0.0
        jobs = _scan_jobs("half_kick", 1, case["ions"], seed)
        return {"case": case, "eng": eng, "jobs": jobs, "ph": ph, "ions": eng.inject(jobs, ph)}
    if kind == "tandem":
        model = mq.TandemModel(n=case["tracks"], seed=486 + 1000003 * int(seed), fine=case["fine"], channel=_fields("s14", 0.1), precision=_precision(case))
        return {"case": case, "model": model, "pulse": model.tracks.copy()}
    rng = np.random.default_rng(int(seed))
    nxy = int(round(16.0 / case["h"]))
    # rod positions off by some hundredths of a millimetre, and by some ten-thousandths per mm of length
    mis = [[float(a), float(b), float(c), float(d)] for a, b, c, d in rng.normal(0.0, 1.0, (4, 4)) * [0.03, 0.03, 3e-4, 3e-4]]
    return {"case": case, "geom": mq.Geom(h_mm=case["h"], n_xy=nxy, mis=mis), "bases": [0, 1, 3, 4][:case["bases"]]}


def _ion_arrays(ions):
    # unsigned fields as signed ones of the same bits
    return {k: (v.view("i%d" % v.itemsize) if v.dtype.kind == "u" else v) for k, v in ((k, getattr(ions, k)) for k in (
        "x", "y", "z", "vx", "vy", "vz", "ph_rf", "ph_ac", "rng", "steps", "ncoll", "leg", "status", "jid"))}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        if case["want"] == "sweep":
            p = state["preset"]
            view = mq.sweep.run_sweep(state["eng"], p.species, state["cfg"], p.v_rf, p.v_ac, p.dc(), state["ph"], state["seed"])
            return {"counts": view.counts}
        if case["want"] == "ions":
            ions, _ = state["eng"].run_batch_ions(state["jobs"], state["dc"], state["ph"])
            return _ion_arrays(ions)
        out = state["eng"].run_batch(state["jobs"], state["dc"], state["ph"])
        return {k: (getattr(out, k).view("i8") if k in COUNTS else getattr(out, k)) for k in COUNTS + MEANS}
    if kind == "states":
        ions = state["ions"].copy()
        state["eng"].run_ions(state["jobs"], state["ph"], ions, max_more=case["steps"])
        return _ion_arrays(ions)
    if kind == "tandem":
        m = state["model"]
        # the same pulse again, from step 0 and with clear counters
        m.tracks.copy_from(state["pulse"])
        m.step = 0
        m.counts = type(m.counts)()
        m.advance(case["steps"])
        t = m.tracks
        return {"x": t.x, "y": t.y, "z": t.z, "vx": t.vx, "vy": t.vy, "vz": t.vz, "rng": t.rng.view("i8"), "region": t.region, "last": t.last,
                "ports": m.counts_array().astype(np.int64)}
    f = mq.Fields.build(state["geom"], bases=state["bases"], cache=False, device=0)
    out = {"rf": f.rf, "ac": f.ac}
    out.update({"dc%d" % i: a for i, a in enumerate(f.dc) if a is not None})
    return out


# ---------------------------------------------------------------- what a pass cannot do without

def _nodes(h):
    return int(round(16.0 / h)) ** 2 * int(round(24.2 / h))


def work(case):
    """Bytes: the jobs or states in, the outcomes or states out, and the field nodes (9 floats) the ions can have been at; operations: a
    step combines three fields at eight corners, interpolates three components and updates position and velocity."""
    kind = case["kind"]
    step_flops = 48 * 2 + 21 * 2 + 30
    if kind == "batch":
        steps = MEAN_STEPS[case["physics"]] * case["jobs"] * case["ions"]
        ions = case["jobs"] * case["ions"]
        out = 92 * ions if case["want"] == "ions" else 64 * case["jobs"]
        return {"bytes": 72 * case["jobs"] + out + 36 * min(_nodes(case["h"]), 2 * steps), "flops": step_flops * steps}
    if kind == "states":
        steps = case["ions"] * case["steps"]
        return {"bytes": 2 * 92 * case["ions"] + 36 * min(_nodes(0.1), 2 * steps), "flops": step_flops * steps}
    if kind == "tandem":
        steps = case["tracks"] * case["steps"]
        return {"bytes": 2 * 68 * case["tracks"] + 36 * min(_nodes(0.1), 2 * steps), "flops": step_flops * steps}
    # a multigrid V-cycle and a conjugate-gradient step cost about 60 operations per node, and about 10 of
    # them reach the tolerance; the electrode mask is read, potential and field are written
    n = _nodes(case["h"])
    return {"bytes": case["bases"] * n * (1 + 8 + 8 + 16), "flops": case["bases"] * n * 60 * 10}


# ---------------------------------------------------------------- the same in 64 bits

def exact(case, seed):
    """Collision-free flight has a value that plain 64-bit arithmetic gives: the leap-frog update in the trilinear fields, ion by ion until
    it leaves. Flights with collisions are draws of a random process, whose values only the generator's own stream gives."""
    if case["kind"] != "states" or case["ions"] * case["steps"] > 2e8:
        return None
    st = prepare(case, seed)
    f, ph, job, ions = st["eng"].fields, st["ph"], st["jobs"][0], st["ions"]
    layers = f.geom.layers()
    dev = torch.device("cuda:0")
    dims = (f.nx, f.ny, f.nz)
    rf, ac = (torch.from_numpy(a).to(dev) for a in (f.rf, f.ac))
    dc = torch.zeros(f.n, 3, dtype=torch.float32, device=dev)
    for v, b in zip(FIG4_DC, f.dc):   # the combined field is a 32-bit sum in the order of the bases
        if b is not None:
            dc = dc + torch.tensor(v, dtype=torch.float32, device=dev) * torch.from_numpy(b).to(dev)[:, :3]
    solid = rf[:, 3] > 0.5
    x = torch.stack([torch.from_numpy(getattr(ions, k)) for k in ("x", "y", "z")], 1).to(dev)
    v = torch.stack([torch.from_numpy(getattr(ions, k)) for k in ("vx", "vy", "vz")], 1).to(dev)
    p_rf, p_ac = (torch.from_numpy(getattr(ions, k)).to(dev) for k in ("ph_rf", "ph_ac"))
    qm = 0.5 * job.sp.z * QE / (job.sp.mass * AMU)
    lim = torch.tensor([(d - 1) * f.h for d in dims], dtype=torch.float64, device=dev)
    top = torch.tensor([d - 2 for d in dims], dtype=torch.int64, device=dev)
    stride = torch.tensor([1, f.nx, f.nx * f.ny], dtype=torch.int64, device=dev)
    alive = torch.ones(len(x), dtype=torch.bool, device=dev)
    for n in range(case["steps"]):
        a_rf = job.drive.v_rf * torch.sin(2 * math.pi * torch.frac(p_rf + n * (job.drive.f_rf * ph.dt)))
        a_ac = job.drive.v_ac * torch.sin(2 * math.pi * torch.frac(p_ac + n * (job.drive.f_ac * ph.dt)))
        g = x / f.h
        cell = torch.minimum(g.floor().long().clamp(min=0), top)
        t = g - cell
        e = torch.zeros_like(x)
        for c in range(8):
            o = torch.tensor([c & 1, (c >> 1) & 1, c >> 2], dtype=torch.int64, device=dev)
            q = ((cell + o) * stride).sum(1)
            w = torch.where(o.bool(), t, 1 - t).prod(1)
            field = a_rf[:, None] * rf[q, :3].double() + a_ac[:, None] * ac[q, :3].double() + dc[q].double()
            e += w[:, None] * field
        nv = v + qm * ph.dt * e
        nx = x + nv * ph.dt
        v = torch.where(alive[:, None], nv, v)
        x = torch.where(alive[:, None], nx, x)
        z = x[:, 2]
        node = torch.minimum((x / f.h + 0.5).floor().long().clamp(min=0), top + 1)
        gone = (z > layers[4] * 1e-3) | (z < 0.5e-3) | (x < 0).any(1) | (x > lim).any(1) | solid[(node * stride).sum(1)]
        alive = alive & ~gone
    out = {k: x[:, i] for i, k in enumerate(("x", "y", "z"))}
    out.update({k: v[:, i] for i, k in enumerate(("vx", "vy", "vz"))})
    out.update({"ph_rf": p_rf, "ph_ac": p_ac, "rng": None, "steps": None, "ncoll": None, "leg": None, "status": None, "jid": None})
    return out
