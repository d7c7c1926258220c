"""Performance cases: the work a user of the library has it do, through its
public entry points (``binarytpm_gb300.lib`` and the C ABI behind it).

Each case names its ``kind``:

``thermal``      revolutions of one or several solves of one shape, advanced
                 together, and their surface temperatures read back: the
                 thermal-inertia sweep that every fit consists of.  FAST is the
                 production precision, REFERENCE the bit-exact drop-in, FP64
                 the accuracy check.
``setup``        geometry, shadowing and scattered sunlight of a shape: once
                 per shape, pole and orbital position.
``job``          the whole stage from host arrays: solve, geometry, shadows,
                 scattering, clones, revolutions, temperatures back.
``visibility``   all-pairs visibility toward an observer (Visibility stage).
``viewfactors``  the view-factor lists of a shape (Shape_Selfheating stage).
``crater``       surface roughness: craters of 100 sub-facets on a part of a
                 shape, with or without their forcing.
``flux``         disk-integrated flux at the WISE wavelengths (Observe stage),
                 smooth or rough.

Shapes are seeded icospheres with radial noise: the benchmark's recursive ones
where the frequency is a power of two (20 f^2 facets; f = 8 is 1,280, f = 32
is 20,480), geodesic ones of any other frequency (ragged facet counts).
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from binarytpm_gb300 import lib, mesh, problem

SIGMA = 5.67e-8
AU_KM = 149.6e6
OBSERVER = (1.2, 0.10, 0.35)                # AU, ecliptic latitude and longitude (rad)
WISE_UM = (4.6028, 11.0984, 22.6405)        # the Observe stage's wavelengths
NSF = 100                                   # sub-facets of the crater model
PRECISION = {"fast": lib.FAST, "reference": lib.REFERENCE, "fp64": lib.FP64}


def listed():
    return [
        # the benchmark's sweep: eight thermal inertias of the 21,760-facet binary through the revolutions
        # before the first convergence test, where every facet is active
        _thermal("sweep8_binary_fast", "fast", 32, 8, 56, 720, 8, 6),
        # a smaller sweep solved to convergence: late revolutions with few active facets
        _thermal("converge4_binary_fast", "fast", 16, 8, 56, 720, 4, 301),
        # one single body, the smallest production solve: latency and launches
        _thermal("single_body_fast", "fast", 8, 0, 56, 720, 1, 12),
        # the bit-exact drop-in on a binary of ragged facet counts (5,780 + 500)
        _thermal("binary_reference", "reference", 17, 5, 48, 613, 1, 8),
        # the FP64 accuracy check of a small body (980 facets)
        _thermal("single_body_fp64", "fp64", 7, 0, 32, 360, 1, 4),
        # forcing of a binary in the drop-in's precision (Gauss-Seidel scattering in facet order)
        {"name": "setup_reference", "kind": "setup", "precision": "reference", "primary": 16, "secondary": 4,
         "ntau": 720},
        # the whole Thermal stage for the binary, host arrays in, eight inertias' temperatures out
        {"name": "job_binary_fast", "kind": "job", "precision": "fast", "primary": 32, "secondary": 8, "nx": 56,
         "ntau": 720, "solves": 8, "revs": 6},
        # which facets an observer sees over a rotation of the binary
        {"name": "visibility_binary", "kind": "visibility", "precision": "fast", "primary": 32, "secondary": 8,
         "ntau": 720},
        # view-factor lists of a new shape model
        {"name": "viewfactors_binary", "kind": "viewfactors", "primary": 16, "secondary": 8, "refine": True},
        # roughness of a part of 640 facets: crater revolutions of the production precision
        {"name": "crater_revolutions_fast", "kind": "crater", "precision": "fast", "primary": 8, "secondary": 4,
         "part": 640, "nx": 48, "ntau": 720, "setup": False, "revs": 8},
        # the drop-in's whole roughness stage of a part of 160 facets: forcing, partial shadows, scattering, heating
        {"name": "crater_stage_reference", "kind": "crater", "precision": "reference", "primary": 8, "secondary": 4,
         "part": 160, "nx": 32, "ntau": 360, "setup": True, "revs": 2},
        # the light curve of the binary from its surface temperatures
        {"name": "flux_binary", "kind": "flux", "precision": "reference", "primary": 32, "secondary": 8, "ntau": 720,
         "rough": False},
    ]


def _thermal(name, precision, primary, secondary, nx, ntau, solves, revs, turns=1):
    return {"name": name, "kind": "thermal", "precision": precision, "primary": primary, "secondary": secondary,
            "nx": nx, "ntau": ntau, "solves": solves, "revs": revs, "turns": turns}


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def _grid(rng, turns=1):
    """Depth intervals and steps the explicit scheme is stable for."""
    nx = rng.choice([n for n in (16, 24, 32, 40, 48, 56) if turns * 2 * math.pi * (n / 8) ** 2 / 0.5 < 720])
    least = int(turns * 2 * math.pi * (nx / 8) ** 2 / 0.48) + 1
    return nx, rng.randint(max(96, least), 720)


def draw(rng):
    kind = rng.choice(["thermal", "thermal", "thermal", "thermal", "setup", "job", "visibility", "viewfactors",
                       "crater", "crater", "flux"])
    secondary = rng.choice([0, rng.randint(2, 8), rng.randint(3, 8)])
    if kind == "thermal":
        precision = rng.choice(["fast", "fast", "fast", "reference", "fp64"])
        turns = rng.choice([1, 1, 1, 3]) if secondary else 1
        nx, ntau = _grid(rng, turns)
        most = {"fast": 28, "reference": 16, "fp64": 9}[precision]
        solves = rng.randint(1, 6 if precision == "fast" else 2)
        revs = rng.randint(2, 9)
        if precision == "fast":
            revs = rng.choice([2, 3, 4, 6, 6, rng.randint(7, 12), rng.randint(7, 40)])
        c = _thermal("", precision, _log_int(rng, 4, most), secondary, nx, ntau, solves, revs, turns)
        del c["name"]
        return c
    if kind == "setup":
        precision = rng.choice(["fast", "fast", "reference"])
        return {"kind": kind, "precision": precision, "secondary": secondary, "ntau": rng.randint(96, 720),
                "primary": _log_int(rng, 4, 28 if precision == "fast" else 15)}
    if kind == "job":
        nx, ntau = _grid(rng)
        return {"kind": kind, "precision": "fast", "primary": _log_int(rng, 4, 24), "secondary": secondary, "nx": nx,
                "ntau": ntau, "solves": rng.randint(1, 8), "revs": rng.choice([2, 3, 4, 6])}
    if kind == "visibility":
        return {"kind": kind, "precision": rng.choice(["fast", "reference"]), "primary": _log_int(rng, 4, 28),
                "secondary": secondary, "ntau": rng.randint(96, 720)}
    if kind == "viewfactors":
        return {"kind": kind, "primary": _log_int(rng, 4, 15), "secondary": secondary, "refine": rng.random() < 0.7}
    if kind == "crater":
        nx, ntau = _grid(rng)
        primary = rng.randint(6, 10)
        precision = rng.choice(["fast", "fast", "reference"])
        setup = rng.random() < 0.5
        return {"kind": kind, "precision": precision, "primary": primary, "secondary": secondary,
                "part": _log_int(rng, 20, 200 if setup or precision == "reference" else 500), "nx": nx, "ntau": ntau,
                "setup": setup, "revs": rng.randint(1, 8)}
    rough = rng.random() < 0.4
    return {"kind": kind, "precision": "reference", "primary": _log_int(rng, 4, 6 if rough else 28),
            "secondary": 0 if rough else secondary, "ntau": rng.randint(96, 360 if rough else 720), "rough": rough}


# ------------------------------------------------------------------ shapes
@functools.lru_cache(maxsize=None)
def _sphere(freq):
    """Unit icosphere of 20 freq^2 outward facets: recursive order for a power
    of two, face by face and row by row otherwise."""
    if freq & (freq - 1) == 0:
        return mesh.icosphere(freq.bit_length() - 1)
    v0, f0 = mesh.icosphere(0)
    i, j = np.meshgrid(np.arange(freq + 1), np.arange(freq + 1), indexing="ij")
    keep = i + j <= freq
    bary = np.stack([freq - i[keep] - j[keep], i[keep], j[keep]], 1)
    at = -np.ones((freq + 2, freq + 2), np.int64)
    at[bary[:, 1], bary[:, 2]] = np.arange(len(bary))
    tris = [(at[a, b], at[a + 1, b], at[a, b + 1]) for a in range(freq) for b in range(freq - a)]
    tris += [(at[a + 1, b], at[a + 1, b + 1], at[a, b + 1]) for a in range(freq) for b in range(freq - a - 1)]
    points = np.concatenate([bary @ v0[t] / freq for t in f0])
    faces = np.concatenate([np.array(tris) + k * len(bary) for k in range(len(f0))])
    _, first, inverse = np.unique(np.round(points, 9), axis=0, return_index=True, return_inverse=True)
    v = points[first]
    return v / np.linalg.norm(v, axis=1, keepdims=True), inverse.reshape(-1)[faces]


def _body(freq, radius_km, noise, seed):
    u, f = _sphere(freq)
    r = np.random.default_rng(seed).uniform(-noise, noise, len(u))
    total, count = np.zeros(len(u)), np.zeros(len(u))
    for a, b in ((0, 1), (1, 2), (2, 0)):  # one Laplacian pass: every edge is seen from both sides
        np.add.at(total, f[:, a], r[f[:, b]])
        np.add.at(count, f[:, a], 1.0)
    r = radius_km * (1.0 + 0.5 * r + 0.5 * total / count)
    return u * r[:, None], f


def _mesh(case, seed):
    v, f = _body(case["primary"], 0.39, 0.05, seed)
    split = len(v), len(f)
    if case["secondary"]:
        v, f = mesh.binary_system((v, f), _body(case["secondary"], 0.08, 0.08, seed + 100003), 1.19)
    return np.ascontiguousarray(v), np.ascontiguousarray(f, np.int32), split


@functools.lru_cache(maxsize=1)
def _context():
    return lib.Context(0)


def _problem(case, seed, lists=True):
    v, f, split = _mesh(case, seed)
    if lists:
        ptr, idx, vf, vec, _ = lib.viewfactors(_context(), v, f, refine=True)
        if case["kind"] == "crater":
            ptr, idx, vf, vec = _without_grazing(v, f, ptr, idx, vf, vec)
    else:
        ptr, idx, vf = problem.empty_lists(len(f))
        vec = np.zeros((0, 3), np.float32)
    return problem.Problem(vertices=v, facets=f, dep_ptr=ptr, dep_idx=idx, dep_vf=vf, ntau=case["ntau"],
                           nx=case.get("nx", 16), polar=(1.0, 0.0, 0.0), pole=problem.BINARY_POLE,
                           rotation_period_s=(11.9 if case["secondary"] else 2.26) * 3600.0, albedo=0.02,
                           emissivity=0.9, tacc=0.005, meta={"dep_vec": vec, "split": split})


def _without_grazing(v, f, ptr, idx, vf, vec):
    """The lists less the entries within 1e-3 of the facet's own plane: the
    crater stage divides by their direction's normal component."""
    n = np.cross(v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]])
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    rows = np.repeat(np.arange(len(f)), np.diff(ptr))
    keep = (vec * n[rows]).sum(1) > 1e-3 * np.linalg.norm(vec.astype(np.float64), axis=1)
    count = np.bincount(rows[keep], minlength=len(f))
    return np.concatenate([[0], np.cumsum(count)]).astype(np.int32), idx[keep], vf[keep], vec[keep]


def _inertias(n, seed):
    rng = np.random.default_rng(seed + 7)
    return [200.0] if n == 1 else [float(t) for t in np.geomspace(25.0, 2000.0, n) * rng.uniform(0.9, 1.1, n)]


def _forcing(case, prob):
    """Shadows and (singly) scattered sunlight in the bit-exact precision: a
    user keeps them from one thermal run for the next."""
    s = _turning(case, lib.Solve(_context(), prob.with_(multiple_scattering=0), precision=lib.REFERENCE))
    s.geometry_shadow()
    s.scattering()
    out = s.shadow(), s.illumination()
    s.close()
    return out


def _turning(case, solve):
    if case.get("turns", 1) != 1:  # a non-synchronous binary: the primary turns more often
        solve.set_binary_rotation(*solve.problem.meta["split"], case["turns"], 1)
    return solve


# ------------------------------------------------------------- crater model
@functools.lru_cache(maxsize=1)
def _crater_model():
    """A hemispherical crater of rim radius 10: 61 vertices, 100 sub-facets
    and the view factors of a sphere's inside (A_j / 4 pi R^2, all pairs)."""
    rings, v, start = 5, [(0.0, 0.0, -10.0)], [0]
    for k in range(1, rings + 1):
        start.append(len(v))
        polar = 0.5 * math.pi * k / rings
        for m in range(4 * k):
            az = 0.5 * math.pi * m / k
            v.append((10 * math.sin(polar) * math.cos(az), 10 * math.sin(polar) * math.sin(az), -10 * math.cos(polar)))
    f = []
    for k in range(1, rings + 1):
        inner, outer = start[k - 1], start[k]
        n_in, n_out = max(1, 4 * (k - 1)), 4 * k
        for q in range(4):
            for m in range(k):
                a, b = outer + (q * k + m) % n_out, outer + (q * k + m + 1) % n_out
                f.append((inner + (q * (k - 1) + m) % n_in, a, b))
            for m in range(k - 1):
                f.append((inner + (q * (k - 1) + m) % n_in, outer + (q * k + m + 1) % n_out,
                          inner + (q * (k - 1) + m + 1) % n_in))
    v, f = np.array(v, np.float32), np.array(f, np.int32)
    n = np.cross(v[f[:, 1]] - v[f[:, 0]], v[f[:, 2]] - v[f[:, 0]])
    flip = (n * v[f].mean(1)).sum(1) > 0  # normals point into the bowl
    f[flip] = f[flip][:, [0, 2, 1]]
    area = 0.5 * np.linalg.norm(n, axis=1)
    vf = np.tile(area[None, :] / (4 * math.pi * 100.0), (NSF, 1)).astype(np.float32)
    np.fill_diagonal(vf, 0.0)
    return v, f, vf


def _check(rc):
    if rc:
        raise lib.AtpmError(rc, lib.load().atpm_last_error().decode(errors="replace"))


def _crater_forcing(state):
    c, s, prob = state["crater"], state["solve"], state["problem"]
    c.prepare_part(s, state["first"], 0, c.nf, prob.meta["dep_vec"])
    c.partial_shadow()
    c.scattering(state["solar"], prob.scattering_accuracy, multiple=True)


# ----------------------------------------------------------------- prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind == "viewfactors":
        v, f, _ = _mesh(case, seed)
        # room for the lists, as a caller of the C interface keeps it from shape to shape
        p, q = 20 * case["primary"] ** 2, 20 * case["secondary"] ** 2
        room = 4096 + 32 * len(f) + p * q // 2
        return {"kind": kind, "vertices": v.astype(np.float32), "facets": f, "refine": case["refine"],
                "ptr": np.zeros(len(f) + 1, np.int32), "photo": np.zeros((len(f), 3), np.float32),
                "idx": np.zeros(room, np.int32), "vf": np.zeros(room, np.float32),
                "vec": np.zeros((room, 3), np.float32)}
    prob = _problem(case, seed, lists=kind not in ("visibility", "flux"))
    precision = PRECISION[case["precision"]]
    state = {"kind": kind, "problem": prob}
    if kind == "thermal":
        tis = _inertias(case["solves"], seed)
        first = _turning(case, lib.Solve(_context(), prob, precision=precision, revcap=case["revs"]))
        first.set_forcing(*_forcing(case, prob))
        solves = [first] + [first.clone() for _ in tis[1:]]
        return state | {"solves": solves, "tis": tis, "out": _buffers(prob, len(tis))}
    if kind == "setup":
        return state | {"solve": lib.Solve(_context(), prob, precision=precision)}
    if kind == "job":
        for key in ("vertices", "facets", "dep_ptr", "dep_idx", "dep_vf"):
            setattr(prob, key, lib.pinned_copy(getattr(prob, key)))
        return state | {"tis": _inertias(case["solves"], seed), "revs": case["revs"], "precision": precision,
                        "out": _buffers(prob, case["solves"])}
    if kind == "visibility":
        return state | {"solve": lib.Solve(_context(), prob.with_(polar=OBSERVER, shadowing=2), precision=precision)}
    if kind == "flux":
        return state | _prepare_flux(case, seed, prob, precision)
    return state | _prepare_crater(case, seed, prob, precision)


def _buffers(prob, n):
    return [lib.host_buffer((prob.nf, prob.ntau), np.float32) for _ in range(n)]


def _warm_solve(prob, precision, ti=200.0):
    s = lib.Solve(_context(), prob.with_(multiple_scattering=0), precision=precision, revcap=2)
    s.geometry_shadow()
    s.scattering()
    s.set_thermal_inertia(ti)
    s.initialise_temperatures()
    s.run()
    return s


def _prepare_flux(case, seed, prob, precision):
    solve = _warm_solve(prob, precision)
    if not case["rough"]:
        return {"solve": solve, "visible": solve.shadow()}
    # sub-facet temperatures and visible fractions (hundredths), as the roughness stages leave them
    g = torch.Generator("cuda").manual_seed(seed)
    shape = (prob.nf, prob.ntau, NSF)
    t = torch.empty(shape, device="cuda").uniform_(80.0, 400.0, generator=g)
    seen = torch.randint(-40, 101, shape, device="cuda", generator=g).clamp_(min=0).float() / 100
    temperatures = lib.Crater(_context(), prob.nf, prob.ntau, 8, NSF, precision)
    temperatures.set_temperatures(t.cpu().numpy())
    visible = lib.Crater(_context(), prob.nf, prob.ntau, 0, NSF, precision)
    visible.set_array(lib.Crater.SFC_SHADOW, seen.cpu().numpy())
    return {"solve": solve, "visible": solve.shadow(), "sub_t": temperatures, "sub_seen": visible}


def _prepare_crater(case, seed, prob, precision):
    part = min(case["part"], prob.nf)
    solve = _warm_solve(prob, lib.REFERENCE)
    crater = lib.Crater(_context(), part, prob.ntau, prob.nx, NSF, precision)
    crater.set_surface(*_crater_model(), prob.rotation_period_s)
    rng = np.random.default_rng(seed)
    albedo = np.full(part, prob.albedo, np.float32)
    inertia = rng.choice([50.0, 200.0, 800.0], part).astype(np.float32)
    crater.set_properties(np.zeros(part, np.uint8), albedo, inertia)
    state = {"solve": solve, "problem": prob, "crater": crater, "solar": solve.solar(), "inertia": inertia,
             "first": (prob.nf - part) // 2, "setup": case["setup"], "revs": case["revs"],
             "converged": np.zeros(part, np.uint8), "out": lib.host_buffer((part, prob.ntau, NSF), np.float32),
             "lit": lib.host_buffer((part, prob.ntau, NSF), np.float32) if case["setup"] else None}
    if not case["setup"]:
        _crater_forcing(state)
    return state


# --------------------------------------------------------------------- run
def run(state):
    return {"thermal": _run_thermal, "setup": _run_setup, "job": _run_job, "visibility": _run_visibility,
            "viewfactors": _run_viewfactors, "crater": _run_crater, "flux": _run_flux}[state["kind"]](state)


def _advance(solves, tis, out):
    for s, ti in zip(solves, tis):
        s.set_thermal_inertia(ti)
        s.initialise_temperatures()
    counts = np.full((len(solves), solves[0].revcap), -1, np.int32)  # -1: no revolution, the solve had converged
    for row, c in zip(counts, lib.batch_run(solves)):
        row[:len(c)] = c
    return {"temperature": lib.result_temperatures(solves, out), "counts": counts}


def _run_thermal(state):
    return _advance(state["solves"], state["tis"], state["out"])


def _run_setup(state):
    s = state["solve"]
    s.geometry_shadow()
    s.scattering()
    return {"shadow": s.shadow(), "illumination": s.illumination()}


def _run_job(state):
    first = lib.Solve(_context(), state["problem"], precision=state["precision"], revcap=state["revs"])
    first.geometry_shadow()
    first.scattering()
    solves = [first] + [first.clone() for _ in state["tis"][1:]]
    out = _advance(solves, state["tis"], state["out"])
    for s in solves:
        s.close()
    return out


def _run_visibility(state):
    state["solve"].geometry_shadow()
    return {"visible": state["solve"].shadow()}


def _run_viewfactors(state):
    so, held, entries = lib.load(), ctypes.c_void_p(), ctypes.c_int64()
    v, f = state["vertices"], state["facets"]
    _check(so.atpm_viewfactors_compute(_context().h, len(v), len(f), v.ctypes.data, f.ctypes.data, int(state["refine"]),
                                       ctypes.byref(held), ctypes.byref(entries)))
    out = [state[k] for k in ("ptr", "idx", "vf", "vec", "photo")]
    try:
        if entries.value > len(state["idx"]):
            raise ValueError("no room for the lists")
        _check(so.atpm_viewfactors_get(held, *(a.ctypes.data for a in out)))
    finally:
        so.atpm_viewfactors_free(held)
    return {"entries": entries.value, "lists": out}


def _run_crater(state):
    c, prob = state["crater"], state["problem"]
    c.set_properties(converged=state["converged"])
    if state["setup"]:
        _crater_forcing(state)
    c.initialise_temperatures(prob.emissivity, SIGMA)
    for rev in range(state["revs"]):
        c.inertia_difference(prob.emissivity, SIGMA, prob.tacc)
        if rev > 5:
            c.update_converged(prob.tacc)
    stride = c.ntau * c.nsf * 4
    _check(lib.load().atpm_crater_get_array_strided(c.h, c.STEMP1, state["out"].ctypes.data, stride))
    got = {"temperature": state["out"], "converged": c.converged()}
    if state["setup"]:
        _check(lib.load().atpm_crater_get_array(c.h, c.ILLUMINATION, state["lit"].ctypes.data))
        got["illumination"] = state["lit"]
    return got


def _run_flux(state):
    s, eps = state["solve"], state["problem"].emissivity
    if "sub_t" in state:
        v, f, _ = _crater_model()
        return s.disk_flux_rough(state["sub_t"], state["sub_seen"], v, f, OBSERVER, WISE_UM, state["visible"], eps)
    return s.disk_flux(OBSERVER, WISE_UM, state["visible"], eps)


# -------------------------------------------------------------------- work
def work(case):
    """Bytes and operations of one pass that no implementation can do without
    (32-bit values; lists counted at the size shapes like these have)."""
    p, q = 20 * case["primary"] ** 2, 20 * case["secondary"] ** 2
    nf, kind = p + q, case["kind"]
    nnz = 4.0 * nf + 0.22 * p * q  # a few neighbours each, and the two bodies' facing halves
    if kind == "viewfactors":
        return {"bytes": 36.0 * nf + 20 * nnz, "flops": 30.0 * nf * nf + 60.0 * nnz * 20}
    cells = float(nf) * case["ntau"]
    setup = 200 * cells + 4 * nnz * case["ntau"]
    if kind == "setup":
        return {"bytes": 8 * cells + 8 * nnz, "flops": setup + 2 * 6 * nnz * case["ntau"]}
    if kind == "visibility":
        return {"bytes": 4 * cells, "flops": 300 * cells}
    if kind == "flux":
        n = NSF if case["rough"] else 1
        return {"bytes": 8 * cells * n, "flops": 150 * cells * n * len(WISE_UM)}
    if kind == "crater":
        cells = float(min(case["part"], nf)) * case["ntau"] * NSF
        step = 4 * case["nx"] + 40 + 2 * NSF
        flops = case["revs"] * step * cells + (cells * (100 * 12 + 5 * 2 * NSF) if case["setup"] else 0)
        return {"bytes": (8 if case["setup"] else 12) * cells, "flops": flops}
    every = case["solves"] * min(case["revs"], 60)  # a solve to convergence: about that many whole revolutions
    flops = every * (cells * (4 * case["nx"] + 40) + 2 * nnz * case["ntau"])
    if kind == "job":
        return {"bytes": 4 * cells * case["solves"] + 8 * nnz, "flops": flops + setup}
    return {"bytes": (4 + 4 * case["solves"]) * cells + 8 * nnz, "flops": flops}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The outputs in 64 bits by torch.  None for what is a decision (flags,
    lists, counts) and for solves to convergence, which take too long."""
    kind = case["kind"]
    if kind in ("viewfactors", "visibility") or case.get("revs", 0) > 12:
        return None
    if kind == "thermal":
        prob = _problem(case, seed)
        lit = torch.from_numpy(_forcing(case, prob)[1]).cuda().double()
        return {"temperature": [_conduct(case, prob, lit, ti) for ti in _inertias(case["solves"], seed)],
                "counts": None}
    if kind == "setup":
        return {"shadow": None, "illumination": _illumination(_problem(case, seed))}
    if kind == "job":
        prob = _problem(case, seed)
        lit = _illumination(prob)
        return {"temperature": [_conduct(case, prob, lit, ti) for ti in _inertias(case["solves"], seed)],
                "counts": None}
    state = prepare(case, seed)
    return _exact_flux(state) if kind == "flux" else _exact_crater(state)


def _matrix(prob):
    return torch.sparse_csr_tensor(torch.from_numpy(prob.dep_ptr).long(), torch.from_numpy(prob.dep_idx).long(),
                                   torch.from_numpy(prob.dep_vf).double(), (prob.nf, prob.nf)).cuda()


def _newton(t0, t1, a, m1, es):
    for _ in range(8):
        t0 = t0 + (a + m1 * (t1 - t0) - es * t0 ** 4) / (m1 + 4 * es * t0 ** 3)
    return t0


def _conduct(case, prob, lit, ti):
    """Revolutions of one solve: [nf][ntau] surface temperatures."""
    nf, ntau, nx = prob.nf, prob.ntau, prob.nx
    es, oma = prob.emissivity * SIGMA, 1.0 - prob.albedo
    turns = torch.ones(nf, dtype=torch.float64, device="cuda")
    if case.get("turns", 1) != 1:
        turns[:prob.meta["split"][1]] = case["turns"]
    dz = 8.0 / nx
    r = (2 * math.pi / ntau / dz ** 2) * turns
    m1 = ti * torch.sqrt(2 * math.pi * turns / prob.rotation_period_s) / dz
    start = (oma * lit.mean(1) / es) ** 0.25
    column = start.repeat(nx + 1, 1)
    old = start[:, None].repeat(1, ntau)
    frozen, m = None, _matrix(prob) if prob.nnz else None
    absorbed = oma * lit.t().contiguous()
    for rev in range(case["revs"]):
        a = absorbed + (m @ (es * old ** 4)).t() if m is not None else absorbed
        new, before = torch.empty(ntau, nf, dtype=torch.float64, device="cuda"), column
        column = column.clone()
        for s in range(ntau):
            column[1:-1] += r * ((column[2:] - 2 * column[1:-1]) + column[:-2])
            column[0] = _newton(column[0], column[1], a[s], m1, es)
            column[-1] = column[-2]
            new[s] = column[0]
        new = new.t().contiguous()
        if frozen is not None:
            new, column = torch.where(frozen[:, None], old, new), torch.where(frozen, before, column)
        if rev > 5:
            still = ((new - old).abs() >= prob.tacc).any(1)
            frozen = ~still if frozen is None else frozen | ~still
        old = new
    return old


def _placed(prob, unit=1.0):
    """Heliocentric vertices [ntau][nv][3]: rotation about the body's axis, the pole's frame, the centre."""
    lat, lon = prob.pole
    sg = math.sin(math.acos(math.cos(lat) * math.sin(abs(lon))))
    cl, sl, co, so = math.cos(lat), math.sin(lat), math.cos(lon), math.sin(lon)
    frame = [[sl / sg, -cl * cl * so * co / sg, cl * co], [0.0, (sl * sl + cl * cl * co * co) / sg, cl * so],
             [-cl * co / sg, -sl * cl * so / sg, sl]]
    a = 2 * math.pi * torch.arange(prob.ntau, dtype=torch.float64, device="cuda")[:, None] / prob.ntau
    x, y, z = torch.from_numpy(prob.vertices).cuda().unbind(1)
    turned = torch.stack([x * torch.cos(a) - y * torch.sin(a), x * torch.sin(a) + y * torch.cos(a),
                          z.expand(prob.ntau, -1)], -1)
    return turned @ torch.tensor(frame, dtype=torch.float64, device="cuda").t() + _cartesian(prob.polar, unit)


def _cartesian(polar, unit):
    d, lat, lon = polar
    return unit * AU_KM * d * torch.tensor([math.cos(lat) * math.cos(lon), math.cos(lat) * math.sin(lon),
                                            math.sin(lat)], dtype=torch.float64, device="cuda")


def _illumination(prob):
    """Sunlight on every facet and step, scattered to the fixed point: [nf][ntau]."""
    solar = 1367.0 / prob.polar[0] ** 2
    f = torch.from_numpy(prob.facets).long().cuda()
    g = torch.repeat_interleave(torch.arange(prob.nf, device="cuda"), torch.from_numpy(np.diff(prob.dep_ptr)).cuda())
    h = torch.from_numpy(prob.dep_idx).long().cuda()
    placed = _placed(prob)
    direct = torch.empty(prob.nf, prob.ntau, dtype=torch.float64, device="cuda")
    for s in range(prob.ntau):
        v = placed[s]
        v0, v1, v2 = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
        mid = (v0 + v1 + v2) / 3
        n = torch.cross(v1 - v0, v2 - v0, dim=1)
        n = n / n.norm(dim=1, keepdim=True)
        dist = mid.norm(dim=1)
        cos = -(n * mid).sum(1) / dist
        lit = cos >= 0
        k = (lit[g] & (dist[g] > dist[h])).nonzero()[:, 0]
        gk, hk = g[k], h[k]
        nh, p0, p1, p2 = n[hk], v0[hk], v1[hk], v2[hk]
        x = mid[gk] * ((mid[hk] * nh).sum(1) / (mid[gk] * nh).sum(1))[:, None]
        inside = torch.ones(len(k), dtype=torch.bool, device="cuda")
        for a, b in ((p0, p1), (p1, p2), (p2, p0)):
            inside &= (torch.cross(b - a, x - a, dim=1) * nh).sum(1) >= 0
        lit[gk[inside]] = False
        direct[:, s] = solar * cos * lit
    if not prob.nnz:
        return direct
    m, lit = _matrix(prob), direct
    for _ in range(12):
        lit = direct + prob.albedo * (m @ lit)
    return lit


def _planck(um, t):
    lam, c, h, k = um * 1e-6, 299792458.0, 6.626068963e-34, 1.380650424e-23
    return 2 * h * c * c / lam ** 5 / torch.expm1(h * c / (lam * k * t))


def _exact_flux(state):
    prob, eps = state["problem"], state["problem"].emissivity
    f = torch.from_numpy(prob.facets).long().cuda()
    temp = torch.from_numpy(state["solve"].surface_temperature64()).cuda()
    seen = torch.from_numpy(state["visible"]).cuda() > 0
    placed = _placed(prob, 1e3)  # the stage's metres around a shape in its own units
    observer = _cartesian(prob.polar, 1e3) - _cartesian(OBSERVER, 1e3)
    rough = "sub_t" in state
    if rough:
        cv, cf, _ = _crater_model()
        c = torch.from_numpy(cv).cuda().double()[torch.from_numpy(cf).long().cuda()]
        cn = torch.cross(c[:, 1] - c[:, 0], c[:, 2] - c[:, 0], dim=1)
        ca = cn.norm(dim=1) / 2
        cn = cn / (2 * ca[:, None])
        sub_t = np.empty((prob.nf, prob.ntau, NSF), np.float32)
        _check(lib.load().atpm_crater_get_array_strided(state["sub_t"].h, 8, sub_t.ctypes.data, prob.ntau * NSF * 4))
        sub_t = torch.from_numpy(sub_t).cuda()
        sub_seen = torch.from_numpy(state["sub_seen"].get_array(lib.Crater.SFC_SHADOW)).cuda()
    out = torch.zeros(prob.ntau, len(WISE_UM), dtype=torch.float64, device="cuda")
    area = None
    for s in range(prob.ntau - 1, -1, -1):  # the areas are the last step's
        v0, v1, v2 = (placed[s][f[:, k]] for k in range(3))
        n = torch.cross(v1 - v0, v2 - v0, dim=1)
        length = n.norm(dim=1, keepdim=True)
        n = n / length
        area = length[:, 0] / 2 if area is None else area
        view = observer - (v0 + v1 + v2) / 3
        d2 = (view * view).sum(1)
        cos = (view * n).sum(1) / d2.sqrt()
        use = seen[:, s] & (cos >= 0)
        for i, um in enumerate(WISE_UM):
            if not rough:
                out[s, i] = (_planck(um, temp[:, s]) * eps * area * cos / d2 * use).sum()
                continue
            edge = (v1 - v0) / (v1 - v0).norm(dim=1, keepdim=True)
            local = torch.stack([(edge * view).sum(1), (torch.cross(n, edge, dim=1) * view).sum(1),
                                 (n * view).sum(1)], 1) / d2.sqrt()[:, None]
            term = _planck(um, sub_t[:, s].double()) * eps * ca * sub_seen[:, s].double() * (local @ cn.t())
            out[s, i] = (term.sum(1) / d2 * area / (ca * cn[:, 2]).sum() * use).sum()
    return out


def _exact_crater(state):
    """The part's sub-facet temperatures from the forcing that the crater holds
    (its partial shadows are decisions, its scattering is not)."""
    c, prob = state["crater"], state["problem"]
    if state["setup"]:
        _crater_forcing(state)
    nf, ntau, nx = c.nf, c.ntau, c.nx
    es, oma, alb, dz = prob.emissivity * SIGMA, 1.0 - prob.albedo, prob.albedo, 8.0 / nx
    vf = torch.from_numpy(_crater_model()[2]).cuda().double()

    def held(which):
        return torch.from_numpy(c.get_array(which)).cuda().double()

    direct = state["solar"] * held(c.SFC_SHADOW) * held(c.SFC_SUN_ANGLE) + held(c.GLOBAL_ILLUMINATION)
    lit = direct
    for _ in range(12):
        lit = direct + alb * (lit @ vf)
    absorbed = oma * lit + held(c.GLOBAL_HEATING)
    start = (absorbed.mean(1) / es) ** 0.25
    start = ((absorbed.mean(1) + (es * start ** 4) @ vf) / es) ** 0.25
    column = start.repeat(nx + 1, 1, 1)
    old = start[:, None].repeat(1, ntau, 1)
    r = 2 * math.pi / ntau / dz ** 2
    inertia = torch.from_numpy(state["inertia"]).cuda().double()
    m1 = (inertia * math.sqrt(2 * math.pi / prob.rotation_period_s) / dz)[:, None]
    for _ in range(state["revs"]):
        a = absorbed + (es * old ** 4) @ vf
        new = torch.empty_like(old)
        for s in range(ntau):
            column[1:-1] += r * ((column[2:] - 2 * column[1:-1]) + column[:-2])
            column[-1] = column[-2]
            column[0] = _newton(column[0], column[1], a[:, s], m1, es)
            new[:, s] = column[0]
        old = new
    got = {"temperature": old, "converged": None}
    if state["setup"]:
        got["illumination"] = lit
    return got
