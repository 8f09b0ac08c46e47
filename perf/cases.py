"""The work that a user's program has this package do, as measurable cases.

Kinds of case (the "kind" value):
  dt      hydro_vnr_dt_noalloc on a state in the caller's device memory: a
          host solver that embeds the CFL time step in its own loop.
  whole   a run from its options to its end: creation (the initial state is
          built on the device), all cycles, the final fields to the host.
          What a job that asks for one result does.
  driver  the same, stopping for an output every `output` of simulated time
          and fetching the variables the command-line driver writes.  What
          every deck of the reference's test suite does.
  steps   a run that is under way (prepared up to cycle `before`), advanced
          by some cycles, its fields to the host: a job between two outputs.
  batch   many runs of uneven sizes advanced together, from their options to
          their fields: a parameter study.
  serve   a stream of requests through the serving loop, all results fetched.

Every call goes through the package's Python classes or the C ABI that they
bind; fields go into buffers that the program keeps, as a C caller's do.
Seeds change the gas constants, the domain and the values; sizes and options
are the case's (batch, serve: of the package's own seeded mixes, "mix").
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

import mahyco_gb300 as M
from mahyco_gb300 import workloads as W

SOD_X, SOD_Y, BISOD_X, BISOD_Y = 4, 5, 15, 16
ADVECTION, SEDOV, TRIPLE, BUBBLE = 18, 1, 13, 14


def listed():
    # options of a case that are not written take _spec()'s values
    return [
        # the smallest embedded time step: launch latency
        {"name": "dt_64x48", "kind": "dt", "nx": 64, "ny": 48},
        # the largest state the entry point accepts, nearly
        {"name": "dt_1024x1000", "kind": "dt", "nx": 1024, "ny": 1000},
        # the reference's one-dimensional deck size, to its final time, with
        # its outputs: thousands of tiny cycles
        {"name": "sod_200x10", "kind": "driver", "scheme": "vnr", "case": SOD_X, "nx": 200, "ny": 10,
         "nbmat": 1, "limiter": "minmod", "cycles": 1400, "output": 0.05},
        # the reference's triple point deck (PenteBorne mixte), cell-centred scheme
        {"name": "triple_70x30", "kind": "driver", "scheme": "euc", "case": TRIPLE, "nx": 70, "ny": 30,
         "nbmat": 3, "limiter": "superBee", "pb": 1, "pb_mixte": 1, "cycles": 850, "output": 0.5},
        # the Lagrange phase alone, the mesh moving, at 8 times the deck size
        {"name": "lagrange_801x41", "kind": "whole", "scheme": "vnr", "case": BISOD_X, "nx": 801, "ny": 41,
         "nbmat": 2, "projection": 0, "pseudo_centree": 1, "cycles": 600},
        # order-3 remap, ordinary size, ragged
        {"name": "sod_o3_403x257", "kind": "whole", "scheme": "vnr", "case": BISOD_X, "nx": 403, "ny": 257,
         "nbmat": 2, "order": 3, "limiter": "minmod", "cycles": 700, "energy_limit": 0.0},
        # the benchmark's large mesh, from its options to its fields: the
        # first cycles of a large run, most of the mesh still at rest
        {"name": "bisod_2048", "kind": "whole", "scheme": "vnr", "case": BISOD_Y, "nx": 2048, "ny": 2048,
         "nbmat": 2, "pb": 1, "variant": 1, "unit": 1, "cycles": 200},
        # the same options on an odd mesh where the whole flow moves
        {"name": "bisod_moving_1001x999", "kind": "steps", "scheme": "vnr", "case": BISOD_Y, "nx": 1001,
         "ny": 999, "nbmat": 2, "pb": 1, "variant": 1, "before": 2600, "cycles": 40,
         "energy_limit": 0.0},
        # the benchmark's three-material triple point, order 3
        {"name": "triple_1792x768", "kind": "whole", "scheme": "euc", "case": TRIPLE, "nx": 1792, "ny": 768,
         "nbmat": 3, "order": 3, "cycles": 60},
        # the triple point under way, order 2 with PenteBorne mixte
        {"name": "triple_moving_641x275", "kind": "steps", "scheme": "euc", "case": TRIPLE, "nx": 641,
         "ny": 275, "nbmat": 3, "limiter": "minmod", "pb": 1, "pb_mixte": 1, "before": 1200, "cycles": 60},
        # a parameter study of the seeded mix (Sod, Sedov, advection)
        {"name": "batch_40", "kind": "batch", "runs": 40, "cycles": 100, "max_nx": 1024, "max_ny": 256,
         "mix": 20261203},
        # requests of all three kinds, 1 to 3 materials
        {"name": "serve_24", "kind": "serve", "runs": 24, "cycles": 150, "max_n": 512, "mix": 107},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dt", "vnr", "vnr", "vnr", "lagrange", "euc", "euc", "batch", "serve"])
    if kind == "dt":
        nx = _log_int(rng, 2, 4000)
        return {"kind": "dt", "nx": nx, "ny": _log_int(rng, 2, min(4000, 1048576 // nx))}
    if kind == "batch":
        return {"kind": "batch", "runs": rng.randint(2, 40), "cycles": rng.randint(20, 100),
                "max_nx": _log_int(rng, 80, 1024), "max_ny": _log_int(rng, 80, 256),
                "mix": rng.randrange(1 << 20)}
    if kind == "serve":
        return {"kind": "serve", "runs": rng.randint(2, 24), "cycles": rng.randint(60, 150),
                "max_n": _log_int(rng, 64, 512), "mix": rng.randrange(1 << 20)}
    c = {"kind": "whole", "scheme": "euc" if kind == "euc" else "vnr"}
    c["nx"], c["ny"] = _log_int(rng, 8, 1500), _log_int(rng, 8, 1500)
    if kind == "euc":
        c["case"] = rng.choice([TRIPLE, TRIPLE, BISOD_X, BUBBLE])
        c["nbmat"] = 3 if c["case"] == TRIPLE else 2
    else:
        c["case"] = rng.choice([SOD_X, SOD_Y, BISOD_X, BISOD_Y, BISOD_Y, ADVECTION])
        c["nbmat"] = 1 if c["case"] in (SOD_X, SOD_Y) else 2
    cost = 2.0 if kind == "euc" else 1.0
    c["cycles"] = max(20, min(600, int(4e7 / (cost * c["nx"] * c["ny"]))))
    if kind != "euc":
        c["energy_limit"] = 0.0
    if kind == "lagrange":
        c["case"], c["nbmat"], c["projection"] = BISOD_X, 2, 0
        c["pseudo_centree"] = rng.randint(0, 1)
        return c
    c["order"] = rng.choice([1, 2, 2, 2, 3])
    c["limiter"] = rng.choice(["minmod", "superBee", "superBee", "vanLeer"])
    if c["order"] == 2 and rng.random() < 0.6:
        c["pb"] = 1
        c["pb_mixte"] = rng.randint(0, 1)
        c["pb_complet"] = rng.choice([0, 0, 1])
        if kind == "vnr":
            c["dual"] = rng.choice([0, 0, 1, 2])
    return c


def _spec(case, rng):
    s = M.default_spec()
    vnr = case["scheme"] == "vnr"
    t = case["case"]
    s.scheme = M.SCHEME_VNR if vnr else M.SCHEME_EUCCLHYD
    s.test_case, s.nbmat = t, case["nbmat"]
    s.nx, s.ny = case["nx"], case["ny"]
    # the domain, a little larger or smaller with the seed (the benchmark's
    # own mesh keeps its unit square)
    k = 1.0 if case.get("unit") else rng.uniform(0.97, 1.03)
    if t == TRIPLE:
        s.dx, s.dy = 7.0 * k / s.nx, 3.0 * k / s.ny
        s.init_variant = 3
    elif t == BUBBLE:
        s.dx, s.dy = 0.65 * k / s.nx, 0.08 * k / s.ny
    else:
        # unit length along the flow; the decks' cells are wider across it
        along, wide = k / (s.ny if t in (SOD_Y, BISOD_Y) else s.nx), 1.0 if case.get("unit") else 1.5
        s.dx, s.dy = (wide * along, along) if t in (SOD_Y, BISOD_Y) else (along, wide * along)
        s.init_variant = case.get("variant", 0)
    g = 1.4 + rng.uniform(-0.03, 0.03)
    for m in range(3):
        s.eos[m] = 101
        s.gamma[m] = g + (0.1 if t == TRIPLE and m != 1 else 0.0)
    s.gamma_scalar, s.cfl = g, 0.4
    s.final_time = s.output_time = 1000.0
    s.dt_init, s.dt_min = 1e-4, 1e-12
    s.space_order = 2
    s.projection, s.projection_order = case.get("projection", 1), case.get("order", 2)
    s.limiter = M.LIMITERS[case.get("limiter", "superBee")]
    s.pb, s.pb_mixte = case.get("pb", 0), case.get("pb_mixte", 0)
    s.limiter_pure, s.pb_complet = M.LIMITERS["arithmeticG"], case.get("pb_complet", 0)
    s.dual_mass_flux = case.get("dual", 0)
    s.pseudo_centree = case.get("pseudo_centree", 0)
    s.energy_limit = case.get("energy_limit", 5.0)
    s.max_cycles = case["before"] + 1000000 if "before" in case else case["cycles"]
    if t == ADVECTION:  # the remap alone: no Lagrange phase, a fixed step
        s.sans_lagrange, s.init_variant, s.dt_init = 1, 2, 0.25 * s.dx
    if "output" in case:
        s.output_time = case["output"]
    return s


FIELDS = {"vnr": ("density", "pressure", "energy", "fracvol_env", "node_velocity"),
          "euc": ("density", "pressure", "energy", "fracvol_env", "cell_velocity")}
DUMPS = {"vnr": ("Pressure", "Density", "Energy", "VitesseX", "VitesseY"),
         "euc": ("Pressure", "Density", "Energy", "VelocityX", "VelocityY")}


def _field_size(spec, name):
    cells, nodes = spec.nx * spec.ny, (spec.nx + 1) * (spec.ny + 1)
    if name in ("node_velocity", "node_coord"):
        return 2 * nodes
    if name.startswith("Vitesse"):
        return nodes
    return 3 * cells if name.endswith("_env") else 2 * cells if name == "cell_velocity" else cells


def _fetch(run, name, out):
    rc = M.lib().hydro_run_fetch(run.h, name.encode(), out.ctypes.data_as(C.POINTER(C.c_double)), out.size)
    if rc:
        raise RuntimeError(M.lib().hydro_last_error().decode())


def _fetch_all(run, buffers):
    for name, out in buffers.items():
        _fetch(run, name, out)


def _buffers(spec, names):
    return {n: np.empty(_field_size(spec, n)) for n in names}


def _study(case, rng):
    """Specs of a batch or a request stream: the package's own seeded mixes."""
    if case["kind"] == "batch":
        inst = W.batch_mix(case["runs"], seed=case["mix"], cycles=case["cycles"],
                           nx_range=(64, case["max_nx"]), ny_range=(64, case["max_ny"]))
    else:
        inst = [r.inst for r in W.request_stream(100.0, case["runs"], seed=case["mix"],
                                                 size_range=(32, case["max_n"]),
                                                 cycle_range=(50, case["cycles"]))]
    specs = [i.spec(M) for i in inst]
    for s in specs:
        k = rng.uniform(0.97, 1.03)
        s.dx, s.dy = k * s.dx, k * s.dy
        s.gamma_scalar += rng.uniform(-0.03, 0.03)
        for m in range(3):
            s.gamma[m] = s.gamma_scalar
        if s.sans_lagrange:
            s.dt_init = 0.25 * s.dx
    return specs


def _dt_state(case, seed):
    """Node velocities and sound speed of a flow part of which is at rest."""
    nx, ny = case["nx"], case["ny"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *shape: torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    y = torch.linspace(0.0, 1.0, ny + 1, device="cuda", dtype=torch.float64)[:, None]
    moving = (y > 0.3).to(torch.float64)
    u = moving * (0.4 * torch.sin(6.0 * y) + 0.05 * rand(ny + 1, nx + 1))
    v = moving * (0.6 * torch.cos(5.0 * y) + 0.05 * rand(ny + 1, nx + 1))
    c = 1.1 + 0.2 * torch.sin(7.0 * y[:ny]) + 0.02 * rand(ny, nx)
    k = 0.9 + 0.2 * random.Random(seed).random()
    return {"u": u.contiguous(), "v": v.contiguous(), "c": c.contiguous(), "dx": k / nx, "dy": k / ny,
            "dt_n": 1.0}


def prepare(case, seed):
    rng = random.Random(seed)
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "dt":
        st.update(_dt_state(case, seed))
        st["out"] = torch.empty(1, device="cuda", dtype=torch.float64)
        f = M.lib().hydro_vnr_dt_noalloc
        f.argtypes = [C.c_int, C.c_int, C.c_double, C.c_double, C.c_void_p, C.c_void_p, C.c_void_p, C.c_double,
                      C.c_void_p, C.c_void_p]
        f.restype = C.c_int
        st["call"] = f
        st["args"] = (case["nx"], case["ny"], st["dx"], st["dy"], st["u"].data_ptr(), st["v"].data_ptr(),
                      st["c"].data_ptr(), st["dt_n"], st["out"].data_ptr(),
                      torch.cuda.current_stream().cuda_stream)
    elif kind in ("batch", "serve"):
        st["ctx"] = M.Context(0)
        st["specs"] = _study(case, rng)
        size = {n: [_field_size(s, n) for s in st["specs"]] for n in FIELDS["vnr"]}
        st["fields"] = {n: np.empty(sum(v)) for n, v in size.items()}
        st["views"] = []
        at = dict.fromkeys(size, 0)
        for r in range(len(st["specs"])):
            st["views"].append({n: st["fields"][n][at[n]:at[n] + size[n][r]] for n in size})
            for n in size:
                at[n] += size[n][r]
        if kind == "serve":
            st["server"] = M.Server(st["ctx"])
    else:
        st["ctx"] = M.default_context()
        st["spec"] = _spec(case, rng)
        names = list(FIELDS[case["scheme"]]) + (["node_coord"] if st["spec"].projection == 0 else [])
        st["fields"] = _buffers(st["spec"], names)
        if kind == "steps":
            st["run"] = M.Run(st["spec"], st["ctx"])
            st["run"].step(case["before"])
    return st


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "dt":
        if state["call"](*state["args"]):
            raise RuntimeError(M.lib().hydro_last_error().decode())
        return state["out"]
    if kind == "steps":
        state["run"].step(case["cycles"])
        _fetch_all(state["run"], state["fields"])
        return {"fields": state["fields"], "cycle": state["run"].time()[2]}
    if kind == "whole":
        r = M.Run(state["spec"], state["ctx"])
        r.simulate()
        _fetch_all(r, state["fields"])
        cycle = r.time()[2]
        r.close()
        return {"fields": state["fields"], "cycle": cycle}
    if kind == "driver":
        s = state["spec"]
        r = M.Run(s, state["ctx"])
        dumps, last, done = [], 0.0, False
        while not done:
            t = r.time()[0]
            if t >= last + s.output_time or t == 0.0:
                dumps.append(_buffers(s, DUMPS[case["scheme"]]))
                _fetch_all(r, dumps[-1])
                last = t
            done, _ = r.step_to_output(1 << 20, last + s.output_time)
        _fetch_all(r, state["fields"])
        cycle = r.time()[2]
        r.close()
        return {"fields": state["fields"], "dumps": {n: np.concatenate([d[n] for d in dumps]) for n in dumps[0]},
                "cycle": cycle}
    if kind == "batch":
        runs = [M.Run(s, state["ctx"]) for s in state["specs"]]
        batch = M.Batch(runs, state["ctx"])
        while batch.step(64):
            pass
        for r, v in zip(runs, state["views"]):
            _fetch_all(r, v)
        cycles = np.array([r.time()[2] for r in runs])
        for r in runs:
            r.close()
        return {"fields": state["fields"], "cycles": cycles}
    server = state["server"]
    ids = [server.submit(s, keep=True) for s in state["specs"]]
    at = {rid: k for k, rid in enumerate(ids)}
    cycles = np.zeros(len(ids), dtype=np.int64)
    ended = 0
    while ended < len(ids):
        d = server.poll(1.0)
        if d is not None:
            cycles[at[d.req_id]] = d.cycles
            ended += 1
    for rid in ids:
        _fetch_all(server.result(rid), state["views"][at[rid]])
        server.release(rid)
    return {"fields": state["fields"], "cycles": cycles}


def _state_planes(spec):
    """Doubles per cell that one cycle has to read and write once: the
    persistent state (density, pressure, energy, pseudo-viscosity, sound
    speed or velocity, divergence, node velocity (2), and per material
    density, energy, pressure, fraction, mass fraction, mass,
    pseudo-viscosity)."""
    return 2 * (10 + 7 * spec.nbmat)


# FP64 additions and products per cell, material and cycle that the scheme's
# formulas have where the flow moves (divisions and roots counted once)
FLOPS = {"vnr": 130, "euc": 200}


def work(case):
    if case["kind"] == "dt":
        nx, ny = case["nx"], case["ny"]
        return {"bytes": 8 * (2 * (nx + 1) * (ny + 1) + nx * ny), "flops": 12 * nx * ny}
    rng = random.Random(1)
    specs = _study(case, rng) if case["kind"] in ("batch", "serve") else [_spec(case, rng)]
    b = f = 0
    for s in specs:
        cycles = case["cycles"] if "before" in case else s.max_cycles
        cells = s.nx * s.ny
        b += 8 * cells * (_state_planes(s) * cycles + 10)
        f += cells * cycles * s.nbmat * (FLOPS["vnr"] if s.scheme == M.SCHEME_VNR else FLOPS["euc"])
    return {"bytes": b, "flops": f}


def exact(case, seed):
    # A simulation's fields have no value beyond the scheme's own in 64 bits,
    # in its order of operations: the outputs are held to the start's.
    if case["kind"] != "dt":
        return None
    st = _dt_state(case, seed)
    speed = torch.sqrt(st["u"] ** 2 + st["v"] ** 2)
    mean = (speed[:-1, :-1] + speed[:-1, 1:] + speed[1:, :-1] + speed[1:, 1:]) * 0.25
    dt = 0.05 * math.sqrt(st["dx"] * st["dy"]) / (mean + st["c"])
    return torch.clamp(dt.min(), max=1.05 * st["dt_n"]).reshape(1)
