"""The work a user of this framework has it do, as cases that can be timed.

A case names one call sequence of the Python binding and its sizes.  The kinds:

  dam, column, footing, rain, slopes
            time steps of a particle system between two outputs: `steps` steps
            (Engine.step), then the state read back into the caller's Particle
            records (Engine.download_particles), as the reference's main loop
            runs between two result files.  The state goes on from pass to pass.
  synth     R realisations of a K-term Karhunen-Loeve field into device memory
            (Engine.kl_synthesize): the Monte Carlo field batch
  field     one K-term field in FP64 into the soil's material records
            (Engine.kl_generate): the field of one realisation
  cells     one correlation-matrix field (Engine.rf_generate, flspv 3)

The scenes, materials and time steps are those of scenes.py and bench.py; the
seed makes what differs between two runs of a user: the particles' deviation
from the lattice and their velocities (a state some steps into a run), the
order of a caller's arrays, and the standard normals of the random fields.
"""
from __future__ import annotations

import functools
import math
import os
import random
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(REPO, "multiphase-sph-solver_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import scenes  # noqa: E402
import sphgpu  # noqa: E402

STEPPED = ("dam", "column", "footing", "rain", "slopes")

# what the result files hold of a particle
STATE = ("xp", "vx", "ax", "ux", "rho", "pre", "prew", "sig", "eps", "adps", "strep", "porosity", "satu", "type")

# subloading Cam-clay of the strip footing's bed
MCC = dict(ramda=0.2, kapa=0.04, zmf=1.2, eps0=0.9, poi=0.3, sme0=50.0e3, ann=1.0, ocr=1.5, e=0.0, fs=1.0)


def listed() -> list:
    return [
        # the smallest call: a 2-D dam break of 1,358 particles, its state
        # wanted after every step (a host program that watches the run)
        {"name": "dam_1k_every_step", "kind": "dam", "dx": 0.02, "width": 0.4, "height": 0.8, "steps": 1,
         "form": "fp64", "flknl": 1, "flbndy": 1},
        # the 2-D dam break at dx = 5 mm (14,978 particles): launch and
        # latency bound
        {"name": "dam_15k", "kind": "dam", "dx": 0.005, "width": 0.4, "height": 0.8, "steps": 100, "form": "fp64",
         "flknl": 1, "flbndy": 1},
        # the 3-D saturated soil column at an odd size (245,012 particles),
        # Yang-Liu kernel, no-slip walls, in the FP32-bulk form
        {"name": "column_245k_bulk32", "kind": "column", "dx": 0.0143, "length": 1.02, "width": 0.5, "height": 0.53,
         "steps": 30, "form": "fp32_bulk", "order": "lattice", "flknl": 2, "flbndy": 13},
        # the ordinary size of a 3-D study (616,184 particles)
        {"name": "column_616k", "kind": "column", "dx": 0.01, "length": 1.0, "width": 0.5, "height": 0.5, "steps": 40,
         "form": "fp64", "order": "lattice", "flknl": 1, "flbndy": 1},
        # the same from a caller whose arrays are in a random order, re-sorted
        # by the engine every 20 steps
        {"name": "column_616k_random_order", "kind": "column", "dx": 0.01, "length": 1.0, "width": 0.5,
         "height": 0.5, "steps": 40, "form": "fp64", "order": "random", "flknl": 1, "flbndy": 1},
        # the largest: the soil column at dx = 5 mm (4,454,314 particles)
        {"name": "column_4m", "kind": "column", "dx": 0.005, "length": 1.0, "width": 0.5, "height": 0.5, "steps": 20,
         "form": "fp64", "order": "lattice", "flknl": 1, "flbndy": 1},
        # a strip footing on a subloading Cam-clay bed, penalty contact
        # (591,964 particles)
        {"name": "footing_592k", "kind": "footing", "dx": 0.08, "contact": 3, "steps": 40, "form": "fp64"},
        # the 3-D rainfall slope, three phases (1,169,092 particles)
        {"name": "rain_slope_1m", "kind": "rain", "dx": 0.1, "steps": 20, "form": "fp64"},
        # 48 uneven 2-D slopes in one batched context
        {"name": "slopes_48", "kind": "slopes", "count": 48, "dx": 0.1, "steps": 40, "form": "fp64"},
        # 32 realisations of a 400-term friction field on the 616,184
        # particles of the soil column
        {"name": "synth_32x400", "kind": "synth", "dx": 0.01, "length": 1.0, "width": 0.5, "height": 0.5, "R": 32,
         "K": 400},
        # one realisation's friction field of the reference's 200 terms, FP64,
        # into the material records of the same particles
        {"name": "field_200", "kind": "field", "dx": 0.01, "length": 1.0, "width": 0.5, "height": 0.5, "K": 200},
        # a correlation-matrix field of 4,830 cells on the 5 m slope
        {"name": "cells_5k", "kind": "cells", "H": 5.0, "dx": 0.1, "cells": 5000},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random) -> dict:
    """One more case of the same kinds and ranges."""
    kind = rng.choice(("dam", "dam", "column", "column", "column", "footing", "rain", "slopes", "synth", "field",
                       "cells"))
    form = rng.choice(("fp64", "fp64", "fp32_bulk"))
    if kind == "dam":
        dx = _log(rng, 0.003, 0.03)
        return {"kind": kind, "dx": round(dx, 5), "width": round(rng.uniform(0.25, 0.6), 3),
                "height": round(rng.uniform(0.4, 0.8), 3), "steps": rng.randint(1, 100), "form": form,
                "flknl": rng.choice((1, 2)), "flbndy": rng.choice((1, 13))}
    if kind == "column":
        dx = _log(rng, 0.0075, 0.05)
        return {"kind": kind, "dx": round(dx, 5), "length": round(rng.uniform(0.6, 1.1), 3),
                "width": round(rng.uniform(0.3, 0.5), 3), "height": round(rng.uniform(0.3, 0.55), 3),
                "steps": rng.randint(20, 60), "form": form, "order": rng.choice(("lattice", "lattice", "random")),
                "flknl": rng.choice((1, 1, 2, 3)), "flbndy": rng.choice((1, 1, 13))}
    if kind == "footing":
        return {"kind": kind, "dx": round(_log(rng, 0.08, 0.25), 4), "contact": rng.choice((1, 2, 3)),
                "steps": rng.randint(20, 40), "form": form}
    if kind == "rain":
        return {"kind": kind, "dx": round(_log(rng, 0.1, 0.3), 4), "steps": rng.randint(10, 30), "form": form}
    if kind == "slopes":
        return {"kind": kind, "count": int(_log(rng, 3, 64)), "dx": round(_log(rng, 0.08, 0.25), 4),
                "steps": rng.randint(20, 60), "form": form}
    if kind == "synth":
        return {"kind": kind, "dx": round(_log(rng, 0.01, 0.05), 5), "length": round(rng.uniform(0.6, 1.1), 3),
                "width": round(rng.uniform(0.3, 0.5), 3), "height": round(rng.uniform(0.3, 0.55), 3),
                "R": 16 * rng.randint(1, 8), "K": 8 * rng.randint(13, 50)}
    if kind == "field":
        return {"kind": kind, "dx": round(_log(rng, 0.01, 0.05), 5), "length": round(rng.uniform(0.6, 1.1), 3),
                "width": round(rng.uniform(0.3, 0.5), 3), "height": round(rng.uniform(0.3, 0.55), 3),
                "K": rng.randint(100, 400)}
    H, dx = round(rng.uniform(3.0, 8.0), 2), round(rng.uniform(0.08, 0.2), 3)
    fewest = 5.0 * H * (1.0 + 0.1 * H) / dx ** 2 / 10.0         # a cell holds at most 39 particles
    return {"kind": "cells", "H": H, "dx": dx, "cells": int(_log(rng, max(600.0, fewest), 13000))}


# --------------------------------------------------------------------------
# scenes (a user's input deck: fixed by the case, kept between two states)

def _column(case) -> scenes.Scene:
    L, W, H = case["length"], case["width"], case["height"]
    return scenes.soil_column_3d(dx=case["dx"], block=(L, W, H), box=(2.0 * L, W, 1.2 * H))


def _slope_heights(count: int, dx: float) -> np.ndarray:
    u = np.random.Generator(np.random.Philox(20261203)).random(count)
    return np.round((5.0 + 7.0 * u) / dx) * dx


def _k0_stress(st, K0: float = 0.3 / 0.7) -> None:
    """A geostatic stress in the bed: rho g depth vertically, K0 of it across."""
    soil, xp = st.fields["type"] == 2, st.fields["xp"]
    top = xp[soil, 1].max() + 0.5 * st.params["dr"]
    sv = -np.asarray(st.soil["dens"]) * 9.81 * (top - xp[:, 1])
    for k, f in ((0, K0), (1, 1.0), (2, K0)):
        st.fields["sig"][soil, k] = f * sv[soil]


def _scene(case) -> scenes.Scene:
    kind = case["kind"]
    if kind == "dam":
        sc = scenes.dam_break_2d(dx=case["dx"], water=(case["width"], case["height"]))
    elif kind in ("column", "synth", "field"):
        sc = _column(case)
    elif kind == "footing":
        sc = scenes.footing(ndim=3, dx=case["dx"], bed=(10.0, 5.0, 5.0), width=2.0, height=0.28, gap=2.0, v=0.01,
                            ss_type=case["contact"], myu=0.3, zeta=0.1, steps=5000, matype=1)
        sc = scenes.set_soil_model(sc, 1, **MCC)
    elif kind == "rain":
        sc = scenes.rain_slope_3d(dx=case["dx"])
    else:
        sc = scenes.slope_2d(H=case["H"], dx=case["dx"])
    for flag in ("flknl", "flbndy"):
        if flag in case:
            sc.flags[flag] = case[flag]
    return sc


class _Deck:
    """Initial state of a case: parameters, Particle records, material records."""


@functools.lru_cache(maxsize=2)
def _deck(key: tuple) -> _Deck:
    case, d = dict(key), _Deck()
    d.scene = d.instances = None
    if case["kind"] == "slopes":
        states = [scenes.initialise(scenes.slope_2d(H=float(h), dx=case["dx"], c=10.0e3, fai=25.0, E=2.0e7))
                  for h in _slope_heights(case["count"], case["dx"])]
        d.params, d.instances, fields, d.fluid, d.soil = sphgpu.batch(states)
        d.rain = None
    else:
        d.scene = _scene(case)
        st = scenes.initialise(d.scene)
        if case["kind"] == "footing":
            _k0_stress(st)
        d.params, fields, d.fluid, d.soil, d.rain = st.params, st.fields, st.fluid, st.soil, st.rain
    d.n, d.nd = int(d.params["ntotal"]), int(d.params["ndim"])
    d.xp, d.type = fields["xp"], fields["type"]
    d.fluid, d.soil = np.ascontiguousarray(d.fluid), np.ascontiguousarray(d.soil)
    d.records = sphgpu.particle_records(fields, d.n).view(_RECORD)
    return d


def _record_dtype() -> np.dtype:
    """Particle as the reference lays it out (xp .. etype of Class_particle.h)."""
    lib, spec = sphgpu.load_library(), {"names": [], "formats": [], "offsets": [], "itemsize": sphgpu.PARTICLE_BYTES}
    off, nc = sphgpu.C.c_size_t(), sphgpu.C.c_int()
    for name in sphgpu.FIELDS:
        lib.sphgpu_particle_layout(name.encode(), sphgpu.C.byref(off), sphgpu.C.byref(nc))
        base = "<i4" if name in sphgpu.INT_FIELDS else "<f8"
        spec["names"].append(name)
        spec["formats"].append(base if nc.value == 1 else (base, (nc.value,)))
        spec["offsets"].append(off.value)
    return np.dtype(spec)


_RECORD = _record_dtype()


def _key(case) -> tuple:
    return tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "form", "order", "R", "K")))


def _disturbed(d: _Deck, seed: int) -> tuple:
    """Positions up to 5% of a spacing off the lattice and velocities of about
    1 cm/s for the particles that move freely (water, soil, air)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    free = torch.from_numpy((d.type >= 1) & (d.type <= 3)).cuda().unsqueeze(1)
    axes = torch.tensor([1.0, 1.0, 1.0 if d.nd == 3 else 0.0], dtype=torch.float64, device="cuda")

    def noise(scale):
        v = torch.randn((d.n, 3), generator=g, dtype=torch.float64, device="cuda").clamp_(-2.5, 2.5)
        return torch.where(free, v.mul_(scale) * axes, 0.0).cpu().numpy()

    return d.xp + noise(0.02 * d.params["dr"]), noise(0.01)


# --------------------------------------------------------------------------

class _State:
    pass


def _field_of(case) -> tuple:
    """The random field of a case: its domain and statistics."""
    sc = _deck(_key(case)).scene
    dom = scenes.kl_domain(sc)
    if case["kind"] == "cells":
        f = dict(no=1, type=2, mean=10.0e3, sd=3.0e3, rl=[6.0, 1.5, 0.0], coe=100.0)     # cohesion, lognormal
    else:
        f = dict(no=0, type=1, mean=30.0, sd=3.0, rl=[0.5, 0.3, 0.2], coe=2.0)         # friction angle, normal
    return dom, f


def _cell_ndx(case, dom) -> float:
    ext = 1.2 * (np.asarray(dom["nb_max"]) - np.asarray(dom["nb_min"]))
    return 1.03 * float(np.sqrt(ext[0] * ext[1] / case["cells"]) / case["dx"])


def prepare(case, seed):
    d, s = _deck(_key(case)), _State()
    s.kind = case["kind"]
    s.engine = sphgpu.Engine(d.params, device=0, instances=d.instances)
    rng = np.random.Generator(np.random.Philox(seed))
    if s.kind in STEPPED:
        xp, vxp = _disturbed(d, seed)
        rec, fluid, soil = d.records, d.fluid, d.soil
        rec["xp"], rec["vxp"] = xp, vxp
        if case.get("order") == "random":
            order = rng.permutation(d.n)
            rec, fluid, soil = rec[order], fluid[order], soil[order]
        s.engine.upload_particles(rec.view(np.uint8))
        s.engine.set_materials(fluid, soil)
        if d.rain is not None:
            s.engine.set_rain(d.rain)
        if case.get("order") == "random":
            s.engine.set_reorder(20)
        if case["form"] == "fp32_bulk":
            s.engine.set_precision(sphgpu.PREC_FP32_BULK)
        s.steps = case["steps"]
        s.records = np.zeros(d.n, _RECORD)
        s.bytes = s.records.view(np.uint8)
        return s
    s.engine.upload_particles(d.records.view(np.uint8))
    s.engine.set_materials(d.fluid, d.soil)
    dom, f = _field_of(case)
    s.domain = sphgpu.kl_domain(dom["nb_min"], dom["nb_max"], dom["soil_max"], dom["water_max"])
    s.field = sphgpu.kl_field(f["no"], f["type"], f["mean"], f["sd"], f["rl"], f["coe"])
    if s.kind == "cells":
        s.flags = sphgpu.rf_flags(_cell_ndx(case, dom), 1)
        s.normals = rng.standard_normal((1, s.engine.rf_cells(s.domain, s.flags)))
    else:
        s.K = case["K"]
        s.normals = rng.standard_normal((case.get("R", 1), s.K))
        if s.kind == "synth":
            s.out = torch.empty((case["R"], d.n), dtype=torch.float32, device="cuda")
    return s


def run(s):
    if s.kind in STEPPED:
        s.engine.step(s.steps)
        s.engine.download_particles(s.bytes)
        return {name: s.records[name] for name in STATE}
    if s.kind == "synth":
        s.engine.kl_synthesize(s.domain, s.field, s.normals, s.out.data_ptr(), s.K)
        return s.out
    if s.kind == "field":
        return s.engine.kl_generate(s.domain, [s.field], s.normals, s.K)
    return s.engine.rf_generate(s.domain, [s.field], s.flags, s.normals)


# --------------------------------------------------------------------------

def work(case) -> dict:
    """Per step and particle each pass of the step reads its own fields once
    and writes its outputs once: 806 bytes in 2-D, 1,870 in 3-D (no neighbour
    list), and about 3,000 / 14,000 FP64 operations; the records' members are
    read back once per pass.  Fields: positions in, values out, the products
    (or eigenfunctions) of the expansion, the factor's n^3 / 3."""
    kind = case["kind"]
    if kind == "slopes":
        dx = case["dx"]
        n = sum(int((6.25 * h + 0.75 * h * h) / dx ** 2 + 3 * (7.25 + 2.0 * h) / dx + 6 * h / dx)
                for h in _slope_heights(case["count"], dx))
        nd = 2
    else:
        sc = _scene(case)
        n, nd = sc.n, sc.ndim
    if kind in STEPPED:
        per, ops = (806.0, 3000.0) if nd == 2 else (1870.0, 14000.0)
        members = sum(nc for name, nc in sphgpu.FIELDS.items() if name != "x")
        return {"bytes": n * (per * case["steps"] + 8.0 * members), "flops": n * ops * case["steps"]}
    if kind == "synth":
        return {"bytes": n * (32.0 + 4.0 * case["R"]), "flops": 2.0 * n * case["K"] * case["R"]}
    if kind == "field":
        return {"bytes": n * (32.0 + 8.0), "flops": 4.0 * n * case["K"]}
    c = float(case["cells"])
    return {"bytes": 8.0 * c * c / 2 + 40.0 * n, "flops": c ** 3 / 3.0 + c * c}


# --------------------------------------------------------------------------
# the values in 64 bits

def exact(case, seed):
    kind = case["kind"]
    if kind == "dam" and case["form"] == "fp64" and case["flknl"] == 1 and case["flbndy"] == 1:
        d = _deck(_key(case))
        return _exact_dam(case, d, seed) if d.n * d.n * case["steps"] <= 2.5e10 else None
    if kind in ("synth", "field"):
        return _exact_kl(case, seed)
    if kind == "cells":
        return _exact_cells(case, seed)
    return None          # elasto-plastic soil: no short plain form


def _exact_kl(case, seed):
    """solve_wi / solve_ramdai / solve_h_3D: H = sum_j sqrt(lambda_j) phi_j xi_j
    over the K largest products of the 1-D eigenvalues."""
    d, K, pi = _deck(_key(case)), case["K"], 3.141592653
    dom, f = _field_of(case)
    lo, hi = np.asarray(dom["nb_min"]), np.asarray(dom["nb_max"])
    a, mid = 0.7 * (hi - lo), 0.5 * (hi + lo)
    w, lam = np.zeros((K, 3)), np.zeros((K, 3))
    i = np.arange(K)
    odd = (i + 1) % 2 == 1
    for ax in range(3):
        l = f["rl"][ax]
        x1 = np.where(odd, i, i + 0.5) * pi / a[ax] + 1.0e-6
        x2 = np.where(odd, i + 0.5, i + 1.0) * pi / a[ax] - 1.0e-6

        def fn(x):
            t = np.tan(x * a[ax])
            return np.where(odd, 2.0 / l - x * t, 2.0 / l * t + x)

        xm, going = 0.5 * (x1 + x2), np.ones(K, bool)
        while going.any():          # the roots as far as the expansion takes them
            f1, fm = fn(x1), fn(xm)
            left = f1 * fm < 0.0
            x2 = np.where(going & left, xm, x2)
            x1 = np.where(going & ~left, xm, x1)
            xm = np.where(going, 0.5 * (x1 + x2), xm)
            going &= np.abs(fm) > 1.0e-6
        w[:, ax], lam[:, ax] = xm, 4.0 * l / (4.0 + xm * xm * l * l)
    # a product among the K largest has at most K products at or above it
    t = [(m, n, k) for m in range(K) for n in range(K // (m + 1)) for k in range(K // ((m + 1) * (n + 1)))]
    t = np.array(t)
    prod = lam[t[:, 0], 0] * lam[t[:, 1], 1] * lam[t[:, 2], 2]
    top = np.argsort(-prod, kind="stable")[:K]
    t, se = t[top], torch.from_numpy(np.sqrt(prod[top])).cuda()
    x = torch.from_numpy(d.xp - mid).cuda()
    phi = torch.ones((K, d.n), dtype=torch.float64, device="cuda")
    for ax in range(3):
        for q in np.unique(t[:, ax]):
            wq = w[q, ax]
            s2 = math.sin(2.0 * wq * a[ax]) / 2.0 / wq
            v = torch.cos(wq * x[:, ax]) / math.sqrt(a[ax] + s2) if q % 2 == 0 else \
                torch.sin(wq * x[:, ax]) / math.sqrt(a[ax] - s2)
            for j in np.flatnonzero(t[:, ax] == q):
                phi[j] *= v
    xi = torch.from_numpy(np.random.Generator(np.random.Philox(seed)).standard_normal((case.get("R", 1), K))).cuda()
    h = (xi * se) @ phi
    out = f["mean"] + (dom["soil_max"] - torch.from_numpy(d.xp[:, 1]).cuda()) * f["coe"] + f["sd"] * h
    return torch.where(torch.from_numpy(d.type == 2).cuda(), out, float("nan"))


def _exact_cells(case, seed):
    """The cells' correlation matrix, its Cholesky factor times the normals,
    and each particle's value from its cell."""
    d = _deck(_key(case))
    dom, f = _field_of(case)
    lo, hi = np.asarray(dom["nb_min"])[:2], np.asarray(dom["nb_max"])[:2]
    ext, dr, e = 1.2 * (hi - lo), d.params["dr"], _cell_ndx(case, dom) * d.params["dr"]
    nc = (ext / e).astype(int) + 1
    base = -(nc * e - ext) / 2.0 + 0.01 * dr + lo - 0.1 * (hi - lo)
    jy, jx = np.divmod(np.arange(nc[0] * nc[1]), nc[0])
    c = torch.from_numpy(np.stack([base[0] + (jx + 0.5) * e, base[1] + (jy + 0.5) * e])).cuda()
    dx, dy = ((c[q].unsqueeze(1) - c[q].unsqueeze(0)).abs_() for q in (0, 1))
    cov = torch.exp(-2.0 * (dx / f["rl"][0] + dy / f["rl"][1]))
    factor, info = torch.linalg.cholesky_ex(cov)
    if int(info) != 0:
        return None
    zeta = np.random.Generator(np.random.Philox(seed)).standard_normal((1, nc[0] * nc[1]))
    z = (factor @ torch.from_numpy(zeta[0]).cuda()).cpu().numpy()
    cell = [np.abs(d.xp[:, q] - base[q]) / e for q in (0, 1)]
    cell = cell[1].astype(int) * nc[0] + cell[0].astype(int)
    soil = d.type == 2
    cell = np.where(soil, cell, 0)
    depth = base[1] + (cell // nc[0] + 0.5) * e
    m = f["mean"] + np.where(dom["soil_max"] > depth, f["coe"] * (dom["soil_max"] - depth), 0.0)
    sd = np.sqrt(np.log(1.0 + (f["sd"] / m) ** 2))
    v = np.exp(np.log(m) - 0.5 * sd * sd + sd * z[cell])
    return np.where(soil, v, np.nan).reshape(1, -1)


def _exact_dam(case, d, seed):
    """The steps of the 2-D dam break (water between resting walls) over dense
    neighbour pairs: continuity, Shepard filter, equation of state, viscous
    stress, momentum, XSPH, wall correction, update."""
    P, n, dev = d.params, d.n, "cuda"
    dr, dt, grav = P["dr"], P["dt"], torch.tensor([P["gx"], P["gy"]], dtype=torch.float64, device=dev)
    xp, vp = (torch.from_numpy(v[:, :2].copy()).to(dev) for v in _disturbed(d, seed))
    get = lambda name: torch.from_numpy(np.ascontiguousarray(d.records[name])).to(dev)  # noqa: E731
    m, rhop, rho, prep, pre = (get(k) for k in ("mass", "rhop", "rho", "prep", "pre"))
    axp, ax = get("axp")[:, :2].clone(), get("ax")[:, :2].clone()
    vx = get("vx")[:, :2].clone()
    water = torch.from_numpy(d.type == 1).to(dev)
    f = {k: torch.from_numpy(np.ascontiguousarray(d.fluid[k])).to(dev) for k in ("dens", "porosity", "vis", "vpu")}
    ux, eps = torch.zeros_like(xp), torch.zeros((n, 6), dtype=torch.float64, device=dev)
    sig, prew = torch.zeros_like(eps), torch.zeros(n, dtype=torch.float64, device=dev)
    a1, tmin, tmax = 0.682092613250980 / dr / dr, P["threshold_min"], P["threshold_max"]
    alpha, beta = P["art_vis"][0]
    w1 = water.unsqueeze(1)

    for _ in range(case["steps"]):
        near = torch.cdist(xp, xp, compute_mode="donot_use_mm_for_euclid_dist") <= 2.0 * dr * (1.0 + 1.0e-12)
        near.fill_diagonal_(False)
        i, j = near.nonzero(as_tuple=True)
        x = xp[i] - xp[j]
        r = x.square().sum(1).sqrt()
        s = r / dr
        inner = s <= 1.0
        W = a1 * torch.where(inner, 0.66666667 - s * s + 0.5 * s ** 3, (2.0 - s) ** 3 / 6.0)
        G = (a1 * torch.where(inner, -2.0 * s + 1.5 * s * s, -0.5 * (2.0 - s) ** 2) / (dr * r)).unsqueeze(1) * x
        keep = s <= 2.0
        W, G = W * keep, G * keep.unsqueeze(1)
        ww, wb, bw = water[i] & water[j], water[i] & ~water[j], ~water[i] & water[j]
        same = water[i] == water[j]

        def total(v, mask):
            v = torch.where(mask if v.dim() == 1 else mask.unsqueeze(1), v, 0.0)
            return torch.zeros((n, *v.shape[1:]), dtype=torch.float64, device=dev).index_add_(0, i, v)

        mj, v = m[j], vp[i] - vp[j]
        rc = rhop + torch.where(water, total(mj * (v * G).sum(1), ww) * dt, 0.0)
        up, down = total(mj * W, same), total(mj / rc[j] * W, same)
        rho = torch.where(down.abs() > 1.0e-7, up / down, rc)
        pre = torch.where(water, prep * ((rho / f["dens"] / f["porosity"]) ** 7 - 1.0) + prep, pre)
        vol = mj / rho[j]
        dv = total((vol.unsqueeze(1) * v).unsqueeze(2).mul(G.unsqueeze(1)).reshape(-1, 4), ww)
        colour = total(vol * W, ww | wb)
        u1, d1 = total(vol * pre[j] * W, bw), total(vol * W, bw)
        prew = torch.where(water, prew, torch.where(d1 != 0.0, u1 / d1, u1))
        tr = dv[:, 0] + dv[:, 3]
        shear = dv[:, 1] + dv[:, 2]
        zero = torch.zeros_like(tr)
        new = torch.stack([dv[:, 0] - tr / 3.0, dv[:, 3] - tr / 3.0, -tr / 3.0], 1)
        eps[:, :3] = torch.where(w1, new, eps[:, :3])
        st = -f["vis"].unsqueeze(1) * torch.stack([2.0 * new[:, 0], 2.0 * new[:, 1], 2.0 * new[:, 2], shear, zero,
                                                   zero], 1)
        st[:, :3] -= pre.unsqueeze(1)
        free = torch.tensor([-1.0, -1.0, -1.0, 0.0, 0.0, 0.0], dtype=torch.float64, device=dev)
        part = ((2.0 * colour - tmin) / (tmax - tmin)).unsqueeze(1)
        st = torch.where((colour < tmin / 2.0).unsqueeze(1), free,
                         torch.where((colour < tmax / 2.0).unsqueeze(1), part * st, st))
        sig = torch.where(w1, st, 0.0)
        own = f["porosity"].unsqueeze(1) * sig / (rho * rho).unsqueeze(1)

        def rows(q):
            return torch.stack([q[:, 0] * G[:, 0] + q[:, 3] * G[:, 1], q[:, 3] * G[:, 0] + q[:, 1] * G[:, 1]], 1)

        acc = grav + total(mj.unsqueeze(1) * rows(own[i] + own[j]), ww)
        approach = (v * x).sum(1)
        mu = dr * approach / (r * r + 0.01 * dr * dr)
        visc = torch.where(approach < 0.0, (-alpha * f["vpu"][i] * mu + beta * mu * mu) / ((rho[i] + rho[j]) * 0.5), 0.0)
        acc = acc - total((mj * visc).unsqueeze(1) * G, ww)
        wall = sig[i] * (1.0 / (rho[j] * rho[j]) + 1.0 / (rho[i] * rho[i])).unsqueeze(1)
        acc = acc + total(mj.unsqueeze(1) * rows(wall), wb)
        ax = torch.where(w1, acc, ax)
        vm = torch.where(w1, vp + 0.5 * (axp + ax) * dt, vx)
        xsph = torch.where(wb, 0.006, P["xsph"][0])
        vn = vm + torch.where(w1, total((xsph * vol * W).unsqueeze(1) * (vm[j] - vm[i]), ww | wb), 0.0)
        hit = (vn[i] * x).sum(1)
        b = torch.clamp(1.0 + 0.3 * dr / (r - 0.3 * dr), max=1.5)
        vn = vn + torch.where(w1, total(((1.0 - b) * hit / (r * r)).unsqueeze(1) * x, wb & (hit < 0.0)), 0.0)
        lo = torch.tensor([P["xmin"], P["ymin"]], dtype=torch.float64, device=dev)
        hi = torch.tensor([P["xmax"], P["ymax"]], dtype=torch.float64, device=dev)
        edge = ((xp - hi >= -0.5 * dr) | (xp - lo <= 0.5 * dr)).any(1, keepdim=True)
        vn = torch.where(w1 & edge, 0.0, vn)
        move = (vn + vp) * dt * 0.5
        xp, ux = torch.where(w1, xp + move, xp), torch.where(w1, ux + move, ux)
        vx, vp, axp = vn, torch.where(w1, vn, vp), torch.where(w1, ax, axp)
        rhop = torch.where(water, rho, rhop)

    wide = lambda q: torch.cat([q, torch.zeros((n, 1), dtype=torch.float64, device=dev)], 1)  # noqa: E731
    out = {name: None for name in STATE}
    out.update(vx=wide(vx), ax=wide(ax), ux=wide(ux), rho=rho, pre=pre, prew=prew, sig=sig, eps=eps)
    out["xp"] = wide(xp)
    return out
