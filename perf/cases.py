"""The engine's workloads as performance cases: what its users have it do, through
storm_b200.engine (Engine.step, Engine.step_host, Server) on the problems of
storm_b200.problems.

A case is a dict of plain values.  `prepare` builds the problem and its handle (for the
host cases also a census), `run` makes one pass.  A pass of the resident cases is what a program does that solves from a
given material state: it hands the engine the state, takes its steps with the census
bank resident on the device, and reads the cells back.  It starts with an empty census,
so every pass is the same work and does not depend on the ones before.

Two steps is as far as two runs can be compared: the device adds tallies in any order,
so temperatures after a step agree to rounding, and the comb's copies of a particle
alone in its cell, ceil(w / (w / n)), can then be n or n + 1; one copy more renumbers
the streams of all packets that follow.  The step's last count of copies is not
returned for the same reason.
"""
import math

import numpy as np

from storm_b200 import _abi as A
from storm_b200 import problems
from storm_b200.engine import Engine, Particles, Server
from storm_b200.units import UNITS

KEV = UNITS["kev_kelvin"]


def listed():
    return [
        # the smallest call: a 100-cell slab with a few thousand packets, one step per material update;
        # launches, synchronisations and short histories count
        dict(name="slab_call", kind="slab", precision=64, n=100, per_cell=5, per_face=2000, nmin=50, steps=1),
        # the plain gray FP64 slab at its stated 1e5 packets and 1e5 census particles per step
        dict(name="slab_fp64", kind="slab", precision=64, n=100, per_cell=50, per_face=50000, nmin=500, steps=2),
        # a problem of the serving stream's middle, alone on the GPU
        dict(name="cube24_fp32", kind="uniform", precision=32, n=24, kappa=300.0, packets=100000, steps=2),
        # the two-material step-opacity cube, Random Walk on, 1e7 packets per step: both forms
        dict(name="cube64_fp32", kind="step", precision=32, n=64, per_cell=3, per_face=450, nmin=20, steps=2),
        dict(name="cube64_fp64", kind="step", precision=64, n=64, per_cell=3, per_face=450, nmin=20, steps=2),
        # multigroup, 64 groups with Planck-sampled emission and multigroup Random Walk: both forms
        dict(name="mg72_fp32", kind="mg", precision=32, n=72, groups=64, per_cell=2, nmin=12, steps=2),
        dict(name="mg40_fp64", kind="mg", precision=64, n=40, groups=64, per_cell=2, nmin=12, steps=2),
        # an odd, ragged multigroup problem whose opacity varies inside the groups: the 30-group,
        # 512-cell Densmore slab at its own packet numbers
        dict(name="densmore_fp64", kind="densmore", precision=64, n=512, per_cell=16, per_face=100, nmin=200, steps=2),
        # gray on a Voronoi mesh with lognormal opacity and temperature
        dict(name="voronoi_fp32", kind="voronoi", precision=32, n=40000, packets=4e6, steps=2),
        dict(name="voronoi_fp64", kind="voronoi", precision=64, n=12000, packets=1.2e6, steps=2),
        # a host program that owns its particles (the serial manager's step): census up, step, census down
        dict(name="host48_fp32", kind="host", precision=32, n=48, per_cell=3, per_face=450, nmin=20, steps=1),
        # the serving loop: independent problems of uneven size sharing the GPU
        dict(name="serve24_fp32", kind="serve", precision=32, count=24, n_lo=16, n_hi=48, p_lo=1e4, p_hi=1e6, steps=2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["slab", "uniform", "step", "step", "mg", "mg", "densmore", "ddmc", "voronoi", "host", "serve"])
    precision = rng.choice([32, 64])
    steps = rng.randint(1, 2)
    if kind == "slab":
        return dict(kind=kind, precision=precision, n=int(_log(rng, 50, 400)), per_cell=int(_log(rng, 5, 60)),
                    per_face=int(_log(rng, 500, 50000)), nmin=int(_log(rng, 50, 500)), steps=steps)
    if kind == "uniform":
        return dict(kind=kind, precision=precision, n=int(_log(rng, 16, 64)), kappa=float(rng.uniform(0.1, 1000.0)),
                    packets=int(_log(rng, 1e4, 3e6)), steps=steps)
    if kind in ("step", "host"):
        n = int(_log(rng, 15, 60 if kind == "step" else 47))
        return dict(kind=kind, precision=precision, n=n, per_cell=rng.randint(1, 4), per_face=rng.randint(50, 450),
                    nmin=rng.randint(5, 20), steps=steps if kind == "step" else 1)
    if kind == "mg":
        return dict(kind=kind, precision=precision, n=int(_log(rng, 11, 70 if precision == 32 else 48)),
                    groups=rng.choice([16, 30, 45, 64]), per_cell=rng.randint(1, 4), nmin=rng.randint(4, 12), steps=steps)
    if kind == "densmore":
        return dict(kind=kind, precision=precision, n=int(_log(rng, 100, 1000)), per_cell=rng.randint(4, 30),
                    per_face=rng.randint(50, 2000), nmin=rng.randint(50, 400), steps=steps)
    if kind == "ddmc":   # the step cube with a scattering half that moves by face leaks
        return dict(kind=kind, precision=precision, n=int(_log(rng, 8, 40)), per_cell=rng.randint(1, 4),
                    per_face=rng.randint(50, 450), nmin=rng.randint(5, 20), steps=steps)
    if kind == "voronoi":
        n = int(_log(rng, 500, 30000 if precision == 32 else 12000))
        return dict(kind=kind, precision=precision, n=n, packets=float(int(n * rng.uniform(10, 100))), steps=steps)
    return dict(kind=kind, precision=precision, count=rng.randint(4, 23), n_lo=16, n_hi=rng.randint(20, 48), p_lo=1e4,
                p_hi=float(int(_log(rng, 5e4, 1e6 if precision == 32 else 3e5))), steps=steps)


def _form(case):
    return A.PRECISION_FP32_TRACK if case["precision"] == 32 else A.PRECISION_FP64


def _heated(p, seed, cold, hot):
    """A seeded, partly heated material: a wave from the hot face at x = 0 to a random
    depth, 10 % cell-to-cell variation, and the energies that go with it."""
    rng = np.random.default_rng(seed)
    x, _, _ = p.cell_centers()
    front = rng.uniform(0.3, 0.6) * p.x_edges[-1]
    shape = np.sqrt(np.sqrt(np.maximum(0.0, 1.0 - x / front)))
    p.temperature = (cold + (hot - cold) * shape) * rng.uniform(0.9, 1.1, p.ncells) * KEV
    p.internal_energy = problems.CV_PER_VOLUME * p.temperature * p.volumes()
    p.cell_internal_energy = p.internal_energy.copy()
    return p


def _problem(case, seed):
    form, kind = _form(case), case["kind"]
    if kind == "slab":
        p = problems.gray_slab(nx=case["n"], new_photons_per_cell=case["per_cell"], face_packets=case["per_face"],
                               comb_nmin=case["nmin"], seed=seed, precision=form)
        return _heated(p, seed, 0.05, 0.8)
    if kind == "uniform":
        p = problems.uniform_cube(n=case["n"], kappa=case["kappa"], packets_per_step=case["packets"], seed=seed,
                                  precision=form)
        return _heated(p, seed, 0.01, 0.6)
    if kind in ("step", "host"):
        p = problems.step_cube(n=case["n"], new_photons_per_cell=case["per_cell"], face_packets=case["per_face"],
                               comb_nmin=case["nmin"], seed=seed, precision=form)
        p.per_cell_segment_counters = False   # as in bench.py; the other cases keep the default counters
        return _heated(p, seed, 0.01, 0.6)
    if kind == "ddmc":
        p = problems.ddmc_cube(n=case["n"], new_photons_per_cell=case["per_cell"], face_packets=case["per_face"],
                               comb_nmin=case["nmin"], seed=seed, precision=form)
        return _heated(p, seed, 0.01, 0.6)
    if kind == "mg":   # initial temperatures uniform in [0.01, 0.1] keV, seeded
        return problems.mg_cube(n=case["n"], groups=case["groups"], new_photons_per_cell=case["per_cell"],
                                comb_nmin=case["nmin"], seed=seed, precision=form)
    if kind == "densmore":
        p = problems.densmore2012(nx=case["n"], new_photons_per_cell=case["per_cell"],
                                  boundary_per_face=case["per_face"], comb_nmin=case["nmin"], seed=seed, precision=form)
        return _heated(p, seed, 0.05, 0.9)
    return problems.voronoi_cube(ncells=case["n"], packets_per_step=case["packets"], seed=seed, precision=form)


def _requests(case, seed):
    """The case's stream of problem sizes, opacities and step counts, each with a material and streams of the seed."""
    mix = problems.serving_mix(case["count"], n_range=(case["n_lo"], case["n_hi"]),
                               packets_range=(case["p_lo"], case["p_hi"]), steps_range=(case["steps"], case["steps"]),
                               precision=_form(case))
    for k, (p, _) in enumerate(mix):
        p.seed = 1000 * seed + k
        _heated(p, p.seed, 0.01, 0.6)
    return mix


_CENSUS = ("x", "y", "z", "vx", "vy", "vz", "weight", "cell")


def prepare(case, seed):
    if case["kind"] == "serve":
        return {"kind": "serve", "server": Server(max_active=6, workers=3), "requests": _requests(case, seed)}
    p = _problem(case, seed)
    state = {"kind": case["kind"], "steps": case["steps"], "engine": Engine(p),
             "material": (p.temperature, p.internal_energy, p.cell_internal_energy)}
    if case["kind"] == "host":
        # the program's own particles: the census of a first step, in page-locked memory
        e = state["engine"]
        e.step()
        n = e.census_count()
        state["census"] = e.census(out=Particles.pinned(n))
        # room for the new census, a size of the case alone (the comb aims at half of it)
        state["out"] = Particles.pinned(2 * int(p.ncells * p.comb_nmin * p.comb_factor))
        for f in _CENSUS:
            getattr(state["out"], f)[:] = 0
    return state


_COUNTS = ("census_in", "emitted_cells", "emitted_faces", "census_out_pre_comb", "segments", "rw_steps",
           "escaped", "cutoff")
_ENERGIES = ("energy_census_in", "energy_emitted", "energy_deposited", "energy_escaped", "energy_census_pre_comb",
             "energy_census_out")


def _result(engine, stats):
    return {"counts": np.array([[s[k] for k in _COUNTS] for s in stats], np.int64),
            "energies": np.array([[s[k] for k in _ENERGIES] for s in stats]),
            "debit": np.array([s["energy_emission_debit"] for s in stats]), "cells": engine.cells()}


def run(state):
    if state["kind"] == "serve":
        server = state["server"]
        tickets = [server.submit(p, steps) for p, steps in state["requests"]]
        server.drain()
        done = {r["ticket"]: r for r in server.poll()}
        return {"segments": np.array([done[t]["segments"] for t in tickets], np.int64),
                "temperature": [done[t]["temperature"] for t in tickets]}
    engine = state["engine"]
    engine.set_cell_state(*state["material"])
    if state["kind"] == "host":
        stats, census = engine.step_host(state["census"], state["out"])
        particles = {f: getattr(state["out"], f) for f in _CENSUS}   # the first len(census) are the census
        return dict(_result(engine, [stats]), count=len(census), census=particles)
    engine.set_census(Particles(0))
    return _result(engine, [engine.step() for _ in range(state["steps"])])


def exact(case, seed):
    """The values of a step that are no sums over random histories, where a pass is one step
    of a gray problem: the opacity, the Fleck factor and the energy the emission takes."""
    if case["kind"] not in ("slab", "uniform", "step", "ddmc", "voronoi") or case["steps"] != 1:
        return None
    p = _problem(case, seed)
    T, vol = p.temperature, p.volumes()
    if case["kind"] == "slab":
        sigma = np.minimum(p.kP0 * (KEV / T) ** p.alpha, p.cap)
    else:
        sigma = p.sigma_a
    a, c = UNITS["arad"], UNITS["clight"]
    fleck = 1.0 / (1.0 + 4.0 * a * T ** 3 * sigma * c * p.dt / p.cv_per_mass)
    return {"counts": None, "energies": None,
            "debit": np.array([math.fsum(fleck * vol * a * T ** 4 * sigma * c * p.dt)]),
            "cells": {"temperature": None, "internal_energy": None, "erad_time_avg": None, "erad_census": None,
                      "sigma_a": sigma, "fleck": fleck, "segments": None}}


# particles' segments per step and floating operations per segment (distance to the faces, the
# collision and the census, attenuation, scatter, tallies and random numbers), by kind
_SEGMENTS = {"slab": 10.0, "uniform": 30.0, "step": 15.0, "mg": 2.5, "densmore": 12.0, "ddmc": 30.0, "voronoi": 15.0,
             "host": 15.0}
_FLOPS = {"slab": 120.0, "uniform": 120.0, "step": 120.0, "mg": 200.0, "densmore": 200.0, "ddmc": 120.0,
          "voronoi": 260.0, "host": 120.0}


def _work(p, kind, steps):
    record = 60.0 if p.precision == A.PRECISION_FP32_TRACK else 84.0
    census = p.ncells * p.comb_nmin * p.comb_factor
    faces = 1 if p.mesh is not None else p.shape[1] * p.shape[2]
    packets = 10.0 * p.ncells * p.new_photons_per_cell + faces * p.faces[0].packets_per_face
    cells = 8.0 * p.ncells * 20
    moved = 2 * census * record + (2 * census * 68.0 if kind == "host" else 0.0)
    return (moved + cells) * steps, (census + packets) * _SEGMENTS[kind] * _FLOPS[kind] * steps


def work(case):
    """One pass: per step the census read and written once and the cells' arrays; the operations of its segments."""
    kind = case["kind"]
    if kind == "serve":
        parts = [_work(p, "uniform", s) for p, s in _requests(case, 1)]
    elif kind == "voronoi":   # sizes alone, without building the mesh
        census, record = case["packets"], 60.0 if case["precision"] == 32 else 84.0
        parts = [((2 * census * record + 8.0 * 40 * case["n"]) * case["steps"],
                  2 * census * _SEGMENTS[kind] * _FLOPS[kind] * case["steps"])]
    else:
        parts = [_work(_problem(case, 1), kind, case["steps"])]
    return {"bytes": float(sum(b for b, _ in parts)), "flops": float(sum(f for _, f in parts))}
