"""Timed cases of the GB/SA framework, through its public entry points.

Each case is one thing a user's program does over and over: a single-point
evaluation with new coordinates, an Energy call, a stretch of MD, a
minimisation, a batch of trial conformations, a burst of requests to the
server.  The systems are the reference-built peptides under tests/golden
(one chain, several chains set on a grid, the first chains of the 16-chain
system), each started from its stored coordinates with a seeded displacement
of every atom.  The pair layout is set (tiles or rows) rather than left to the
autotuner, as a program does that wants the same bits from run to run.

A case is a dict:
  kind     what the pass does (the run_* functions below)
  system   "pep8", "pep64", ... one stored peptide; "amber:3+7" / "opls:0"
           library peptides on a 25 A grid; "grid:k" the first k chains of
           the 16 x 80-residue system
  cutoff   non-bonded cutoff (A); the inner cutoff is 3 A less
  layout   "tiles" or "rows"
  and what the kind needs (steps, members, integrator, jobs).
"""
import ctypes
import functools
import json
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "pd.arcus_b200"))

import pdgpu  # noqa: E402
from pdgpu import _abi as A  # noqa: E402

GOLDEN = os.path.join(ROOT, "tests", "golden")
SINGLE = {"pep8": "pep8_s1", "pep20": "pep20_s2", "pep24": "lcpo_pep24_s5", "pep30": "pep30_s3_rc16",
          "pep64": "c1_pep64_s0"}
LIBRARY = {"amber": "lib16_amber_s3", "opls": "lib16_opls_s4"}
# atoms of the library peptides (draw() picks by size without reading the files)
LIB_ATOMS = {"amber": (384, 612, 1984, 1240, 384, 880, 935, 471, 1662, 413, 804, 1057, 896, 1262, 1806, 2972),
             "opls": (1862, 2367, 2191, 1523, 2317, 2413, 2369, 609, 1327, 1658, 1072, 1216, 1766, 2134, 1658, 822)}
DISPLACEMENT = 0.025  # A per coordinate: thermal for bond-stretch degrees of freedom
ASP = 0.005           # kcal/mol/A^2, the solvation parameter the stored LCPO system carries
INTEGRATORS = {"langevin": A.INTEGRATOR_LANGEVIN, "velocity_verlet": A.INTEGRATOR_VELOCITY_VERLET}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a scoring or embedding loop on a small peptide: latency of one call
        {"name": "forces_pep8", "kind": "forces", "system": "pep8", "cutoff": 12.0, "layout": "tiles"},
        # the ordinary single point: one protein domain's worth of atoms
        {"name": "forces_pep64", "kind": "forces", "system": "pep64", "cutoff": 12.0, "layout": "tiles"},
        # the large single point: the 20,566-atom system at its 16 A cutoff
        {"name": "forces_16x80", "kind": "forces", "system": "grid:16", "cutoff": 16.0, "layout": "tiles"},
        # the Energy protocol (energies only, list rows) on the longest library peptide
        {"name": "energy_pep200", "kind": "energy", "system": "amber:15", "cutoff": 12.0, "layout": "rows"},
        # vacuum force field (bonded + force-switched LJ/Coulomb) on an OPLS peptide
        {"name": "vacuum_opls120", "kind": "vacuum", "system": "opls:0", "cutoff": 12.0, "layout": "rows"},
        # GB/SA with the LCPO surface term, four chains
        {"name": "surface_4x80", "kind": "surface", "system": "grid:4", "cutoff": 12.0, "layout": "tiles"},
        # the plain small MD run: one 64-residue peptide, Langevin
        {"name": "md_pep64", "kind": "md", "system": "pep64", "cutoff": 12.0, "layout": "tiles", "steps": 200,
         "integrator": "langevin"},
        # the large MD run: host state in and out around 50 steps
        {"name": "md_16x80", "kind": "md", "system": "grid:16", "cutoff": 16.0, "layout": "tiles", "steps": 50,
         "integrator": "langevin"},
        # steepest descent on one ordinary peptide (1,662 atoms)
        {"name": "minimise_pep110", "kind": "minimise", "system": "amber:8", "cutoff": 12.0, "layout": "tiles",
         "steps": 100},
        # one Monte Carlo round of trial conformations: 512 peptides at once
        {"name": "trials_512", "kind": "trials", "system": "amber:*", "cutoff": 12.0, "layout": "tiles",
         "members": 512},
        # replicas advanced together: 64 OPLS peptides, 40 steps
        {"name": "batch_md_64", "kind": "batch_md", "system": "opls:*", "cutoff": 12.0, "layout": "tiles",
         "members": 64, "steps": 40, "integrator": "langevin"},
        # a burst of single-point requests of mixed sizes to the server
        {"name": "serve_24", "kind": "serve", "system": "amber:*", "cutoff": 12.0, "layout": "tiles", "jobs": 24},
    ]


def _draw_system(rng, lo, hi):
    """A system of about log-uniform size in [lo, hi] atoms."""
    want = float(np.exp(rng.uniform(np.log(lo), np.log(hi))))
    if want < 370:
        return rng.choice(["pep8", "pep20"])
    if want > 3500 and rng.random() < 0.4:
        return "grid:%d" % max(1, min(16, round(want / 1285.0)))
    lib = rng.choice(["amber", "amber", "opls"])
    sizes, parts, left = LIB_ATOMS[lib], [], want
    while left > 300 and len(parts) < 24:
        fits = [k for k in range(16) if sizes[k] <= 1.15 * left]
        if not fits:
            break
        parts.append(rng.choice(fits))
        left -= sizes[parts[-1]]
    return "%s:%s" % (lib, "+".join(str(k) for k in parts or [0]))


def _atoms(system):
    if system.startswith("grid:"):
        return 1285 * int(system[5:])
    if ":" in system:
        lib, parts = system.split(":")
        return sum(LIB_ATOMS[lib][int(k)] for k in parts.split("+"))
    return {"pep8": 133, "pep20": 318}.get(system, 506)


def draw(rng):
    kind = rng.choice(["forces", "forces", "forces", "energy", "vacuum", "surface", "md", "md", "minimise", "trials",
                       "batch_md", "serve"])
    cutoff = rng.choice([10.0, 12.0, 12.0, 14.0, 16.0])
    c = {"kind": kind, "cutoff": cutoff, "layout": "tiles"}
    if kind == "forces":
        c["system"] = _draw_system(rng, 130, 19000)
        c["layout"] = rng.choice(["tiles", "tiles", "tiles", "rows"])
    elif kind in ("energy", "vacuum"):
        c["system"] = _draw_system(rng, 130, 6000)
        c["layout"] = "rows"
    elif kind == "surface":
        c["system"] = rng.choice(["pep24"] + ["grid:%d" % k for k in range(1, 9)])
    elif kind == "md":
        c["system"] = _draw_system(rng, 130, 15000)
        n = _atoms(c["system"])
        c["steps"] = rng.randrange(20, 60 if n > 4000 else 200)
        c["integrator"] = rng.choice(["langevin", "langevin", "velocity_verlet"])
    elif kind == "minimise":
        c["system"] = _draw_system(rng, 130, 5000)
        c["steps"] = rng.randrange(20, 120)
    elif kind == "trials":
        c["system"], c["members"] = "amber:*", int(np.exp(rng.uniform(np.log(8), np.log(400))))
        c["cutoff"] = rng.choice([10.0, 12.0])
    elif kind == "batch_md":
        c["system"], c["members"] = rng.choice(["opls:*", "amber:*"]), int(np.exp(rng.uniform(np.log(4), np.log(60))))
        c["steps"] = rng.randrange(15, 40)
        c["cutoff"] = rng.choice([10.0, 12.0])
        c["integrator"] = rng.choice(["langevin", "velocity_verlet"])
    else:
        c["system"], c["jobs"] = "amber:*", rng.randrange(4, 32)
        c["cutoff"] = rng.choice([10.0, 12.0])
    return c


# ------------------------------------------------------------------ systems
@functools.lru_cache(maxsize=None)
def _stored(name):
    with np.load(os.path.join(GOLDEN, name + ".npz")) as z:
        return {k: z[k] for k in z.files}


@functools.lru_cache(maxsize=None)
def _member(lib, k):
    pre = "p%02d_" % k
    return {f[len(pre):]: v for f, v in _stored(LIBRARY[lib]).items() if f.startswith(pre)}


TOPOLOGY = ("charge", "radius", "epsilon", "mass", "gb_radius", "is_h", "gb_vj", "gb_terms123")
SURFACE = ("lcpo_radius", "lcpo_p", "lcpo_use")
TERMS = (("bond_ij", ("bond_lk",)), ("angle_iaj", ("angle_kt",)), ("tors_idx", ("tors_terms", "tors_par")),
         ("impr_idx", ("impr_terms", "impr_par")))


def _chains(parts, spacing=25.0):
    """Several peptides as one system, each chain's long axis along z, on a
    square grid in x and y."""
    side = int(np.ceil(np.sqrt(len(parts))))
    out = {k: np.concatenate([p[k] for p in parts]) for k in TOPOLOGY}
    pos, off = [], np.cumsum([0] + [len(p["charge"]) for p in parts])
    for k, p in enumerate(parts):
        x = p["pos"] - p["pos"].mean(axis=0)
        axes = np.linalg.svd(x, full_matrices=False)[2]
        axes = axes * np.sign(axes[np.arange(3), np.abs(axes).argmax(axis=1)])[:, None]
        axes[0] *= np.sign(np.linalg.det(axes))
        pos.append(x @ axes[[1, 2, 0]].T + [(k % side) * spacing, (k // side) * spacing, 0.0])
    out["pos"] = np.concatenate(pos)
    res = np.cumsum([0] + [int(p["ir"].max()) + 1 for p in parts])
    out["ir"] = np.concatenate([p["ir"] + r for p, r in zip(parts, res)]).astype(np.int32)
    for c in ("cov12", "cov13", "cov14"):
        ends = np.cumsum([0] + [int(p[c + "_ptr"][-1]) for p in parts])
        out[c + "_ptr"] = np.concatenate([[0]] + [p[c + "_ptr"][1:] + e for p, e in zip(parts, ends)]).astype(np.int32)
        out[c + "_idx"] = np.concatenate([p[c + "_idx"] + o for p, o in zip(parts, off)]).astype(np.int32)
        if c != "cov14":
            out[c + "_d"] = np.concatenate([p[c + "_d"] for p in parts])
    for idx, values in TERMS:
        out[idx] = np.concatenate([p[idx] + o for p, o in zip(parts, off)]).astype(np.int32)
        for v in values:
            out[v] = np.concatenate([p[v] for p in parts])
    bb = [np.where(p["backbone_ncac"] >= 0, p["backbone_ncac"] + o, -1) for p, o in zip(parts, off)]
    out["backbone_ncac"] = np.concatenate(bb).astype(np.int32)
    out["ff_params"] = parts[0]["ff_params"]
    return out


def _first_chains(a, k):
    """The first k of the 16 chains (80 residues each) of the large system."""
    n = int(np.searchsorted(a["ir"], 80 * k))
    out = {f: a[f][:n] for f in TOPOLOGY + SURFACE + ("ir", "pos")}
    for c in ("cov12", "cov13", "cov14"):
        out[c + "_ptr"] = a[c + "_ptr"][:n + 1]
        m = int(out[c + "_ptr"][-1])
        out[c + "_idx"] = a[c + "_idx"][:m]
        if c != "cov14":
            out[c + "_d"] = a[c + "_d"][:m]
    for idx, values in TERMS:
        keep = (a[idx] < n).all(axis=1)
        for f in (idx,) + values:
            out[f] = a[f][keep]
    out["backbone_ncac"] = a["backbone_ncac"][:80 * k]
    out["ff_params"] = a["ff_params"]
    return out


@functools.lru_cache(maxsize=64)
def _arrays(system):
    if system.startswith("grid:"):
        return _first_chains(_stored("c2_16x80_s2"), int(system[5:]))
    if ":" in system:
        lib, parts = system.split(":")
        parts = [_member(lib, int(k)) for k in parts.split("+")]
        return parts[0] if len(parts) == 1 else _chains(parts)
    return _stored(SINGLE[system])


def _members(case):
    """The library peptides of a batch or a server, in a fixed order."""
    lib = case["system"].split(":")[0]
    return ["%s:%d" % (lib, (7 * k) % 16) for k in range(min(16, case.get("members", 16)))]


def _displaced(system, rng):
    p = _arrays(system)["pos"]
    return np.ascontiguousarray(p + rng.normal(0.0, DISPLACEMENT, p.shape))


@functools.lru_cache(maxsize=None)
def _context():
    return pdgpu.Context(0)


def _workspace(case, system, pos, setup=True):
    """WorkSpace + Forcefield with the case's components and layout."""
    a = dict(_arrays(system), pos=pos)
    a = {k: v for k, v in a.items() if not k.startswith(("f_", "trial_"))}
    ws = pdgpu.WorkSpace(pdgpu.SystemSpec(a), _context())
    ff = pdgpu.Forcefield(ws)
    ff.add(pdgpu.FF_Bonded(ws))
    nb = (pdgpu.FF_NonBonded if case["kind"] == "vacuum" else pdgpu.FF_GeneralizedBorn_Still)(ws)
    nb.Cutoff = nb.VdwCutoff = case["cutoff"]
    nb.InnerCutoff = nb.VdwInnerCutoff = case["cutoff"] - 3.0
    ff.add(nb)
    if case["kind"] == "surface":
        sa = pdgpu.FF_SASA_LCPO(ws)
        sa.GlobalASP = ASP
        ff.add(sa)
        ws.surface = sa
    ff.ensuresetup()
    if setup:
        if case["layout"] == "tiles":
            ws.setPairPath(1)
        else:
            ws.setLanes((8, 8, 8))
    return ws, ff


class State:
    """What a program holds between passes; gives the device memory back."""

    def __init__(self, case):
        self.case, self.owned = case, []

    def own(self, x):
        self.owned.append(x)
        return x

    def __del__(self):
        for x in reversed(self.owned):
            x.close()


def _md_params(case, seed):
    p = A.md_params_default()
    p.Integrator, p.UpdateNList, p.UseGraph = INTEGRATORS[case["integrator"]], 10, 1
    p.Timestep, p.FricCoeff, p.TargetTemp, p.Seed = 1e-15, 1e12, 300.0, seed
    return p


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    st = State(case)
    if case["kind"] in ("trials", "batch_md"):
        names = _members(case)
        ws = {n: st.own(_workspace(case, n, _arrays(n)["pos"], setup=False)[0]) for n in names}
        if case["kind"] == "trials":
            for w in ws.values():
                w.setTorsionMoves()
        order = [names[k % len(names)] for k in range(case["members"])]
        st.batch = st.own(pdgpu.Batch([ws[n] for n in order], _context()))
        st.batch.setPairPath(1)
        st.pos = np.concatenate([_displaced(n, rng) for n in order])
        st.batch.setPositions(st.pos)
        st.batch.setSeeds(rng.integers(1, 1 << 60, len(order), dtype=np.uint64))
        st.batch.calcNewList()
        if case["kind"] == "trials":
            st.batch.saveBasePositions()
        else:
            st.params = _md_params(case, seed)
        st.trial = int(seed) & 0xFFFF
        return st
    if case["kind"] == "serve":
        names = _members(case)
        st.ws = {n: st.own(_workspace(case, n, _arrays(n)["pos"])[0]) for n in names}
        st.server = st.own(pdgpu.Server(_context(), hbm_budget=int(40e9)))
        pick = np.random.default_rng(case["jobs"]).integers(0, len(names), case["jobs"])
        st.requests = [(st.ws[names[k]], _displaced(names[k], rng)) for k in pick]
        st.job = pdgpu.Server.job(pdgpu.Server.ENERGY)
        return st
    st.pos = _displaced(case["system"], rng)
    st.ws, st.ff = _workspace(case, case["system"], st.pos)
    st.own(st.ws)
    st.ws.nlist().calcNewList()
    n = len(st.pos)
    if case["kind"] in ("forces", "md", "minimise"):
        # the buffers of a host program that calls the C interface
        st.forces, st.x, st.v = np.empty((n, 3)), np.empty((n, 3)), np.empty((n, 3))
        st.energies = np.empty(A.ENE_COUNT)
    if case["kind"] == "md":
        st.params = _md_params(case, seed)
        m = np.asarray(_arrays(case["system"])["mass"]).reshape(-1, 1)
        st.v0 = np.ascontiguousarray(rng.normal(0.0, 1.0, (n, 3)) * np.sqrt(1.38065e-23 * 300.0 / m))
    if case["kind"] == "minimise":
        st.params = A.min_params_default()
        st.params.Algorithm, st.params.UpdateNList = A.MIN_STEEPEST_DESCENT, 10
    return st


# ------------------------------------------------------------------ one pass
FIELDS = tuple(pdgpu.Hamiltonian.FIELDS)


def _record(ws):
    return np.array([getattr(ws.ene, k) for k in FIELDS])


def run_forces(st):
    """New coordinates, list, forces and energies, as a C host calls them."""
    L, c, s = A.lib(), st.ws.ctx.ptr, st.ws._device()
    A.check(L.pdgpu_set_positions(c, s, A.dptr(st.pos)))
    A.check(L.pdgpu_nlist_build(c, s))
    A.check(L.pdgpu_calc_forces(c, s))
    A.check(L.pdgpu_get_forces(c, s, A.dptr(st.forces)))
    A.check(L.pdgpu_get_energies(c, s, A.dptr(st.energies), A.ENE_COUNT))
    return {"forces": st.forces, "energies": st.energies}


def run_energy(st):
    pdgpu.Energy(st.ff).run()
    return {"forces": st.ws.cur.f, "energies": _record(st.ws)}


def run_vacuum(st):
    st.ws.nlist().calcNewList()
    st.ff.calcForces()
    return {"forces": st.ws.cur.f, "energies": _record(st.ws)}


def run_surface(st):
    st.ws.nlist().calcNewList()
    st.ff.calcForces()
    sasa, deriv = st.ws.surface.sasa()
    return {"forces": st.ws.cur.f, "energies": _record(st.ws), "sasa": sasa, "deriv": deriv}


def run_md(st):
    L, c, s = A.lib(), st.ws.ctx.ptr, st.ws._device()
    k = st.case["steps"]
    A.check(L.pdgpu_md_run_io(c, s, ctypes.byref(st.params), 0, k, k, A.dptr(st.pos), A.dptr(st.v0), A.dptr(st.x),
                              A.dptr(st.v), A.dptr(st.energies)))
    return {"positions": st.x, "velocities": st.v, "energies": st.energies}


def run_minimise(st):
    L, c, s = A.lib(), st.ws.ctx.ptr, st.ws._device()
    taken = ctypes.c_int32(0)
    A.check(L.pdgpu_set_positions(c, s, A.dptr(st.pos)))
    A.check(L.pdgpu_minimise_run(c, s, ctypes.byref(st.params), st.case["steps"], ctypes.byref(taken)))
    A.check(L.pdgpu_get_positions(c, s, A.dptr(st.x)))
    A.check(L.pdgpu_get_forces(c, s, A.dptr(st.forces)))
    A.check(L.pdgpu_get_energies(c, s, A.dptr(st.energies), A.ENE_COUNT))
    return {"positions": st.x, "forces": st.forces, "energies": st.energies, "steps": int(taken.value)}


def run_trials(st):
    st.batch.perturbTorsions(sigma=np.radians(15.0), trial=st.trial)
    forces, energies = st.batch.evaluate()
    return {"forces": forces, "energies": energies}


def run_batch_md(st):
    st.batch.setPositions(st.pos)
    history = st.batch.runMD(st.params, st.case["steps"], init_velocities=300.0)
    return {"positions": st.batch.positions(), "velocities": st.batch.velocities(), "history": history}


def run_serve(st):
    ids = [st.server.submit(ws, st.job, x) for ws, x in st.requests]
    out = []
    for j in ids:
        A.check(st.server.wait(j, 60.0))
        r = st.server.result(j)
        out.append((r["forces"], r["energies"]))
        st.server.release(j)
    return {"forces": np.concatenate([f for f, _ in out]), "energies": np.array([e for _, e in out])}


def run(st):
    return globals()["run_" + st.case["kind"]](st)


# ------------------------------------------------------------------ work
FLOP_BORN, FLOP_PAIR, FLOP_BONDED = 57, 90, 350  # per directed Still pair, unordered pair, atom
FLOP_LJ, FLOP_ENERGY = 45, 40                    # per unordered pair of the vacuum and energy-only terms
FLOP_SURFACE = 50e3                              # per heavy atom (about 850 overlapping triples at 58 flop)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


@functools.lru_cache(maxsize=None)
def _pairs(system, cutoff):
    """(directed pairs inside the 10 A Still cutoff, unordered pairs inside the cutoff)."""
    x = torch.as_tensor(_arrays(system)["pos"], device=_device())
    still = inside = 0
    for b in range(0, len(x), 1024):
        d2 = (x[b:b + 1024, None, :] - x[None, :, :]).square().sum(-1)
        still += int((d2 <= 100.0).sum())
        inside += int((d2 <= cutoff * cutoff).sum())
    return still - len(x), (inside - len(x)) // 2


def work(case):
    kind, rc = case["kind"], case["cutoff"]
    if kind in ("trials", "batch_md"):
        names = _members(case)
        systems = [names[k % len(names)] for k in range(case["members"])]
    elif kind == "serve":
        names = _members(case)
        systems = [names[k] for k in np.random.default_rng(case["jobs"]).integers(0, len(names), case["jobs"])]
    else:
        systems = [case["system"]]
    n = flops = 0
    for s in systems:
        a = _arrays(s)
        still, inside = _pairs(s, rc)
        n += len(a["charge"])
        flops += FLOP_BONDED * len(a["charge"])
        if kind == "vacuum":
            flops += FLOP_LJ * inside
        elif kind == "energy":
            flops += 21 * still + (FLOP_LJ + FLOP_ENERGY) * inside
        else:
            flops += FLOP_BORN * still + FLOP_PAIR * inside
        if kind == "surface":
            flops += FLOP_SURFACE * int(np.sum(a["lcpo_use"]))
    steps = case.get("steps", 1)
    state = 48 * n  # positions in, forces (or positions) out
    if kind in ("md", "batch_md"):
        state += 48 * n  # velocities in and out
    return {"bytes": float(state), "flops": float(flops * steps)}


# ------------------------------------------------------------------ in 64 bits
KCAL = 4184.0 / 6.0221418e23                                        # kcal/mol in J per molecule
ECONV = (6.0221418e23 / 4184.0) * 1.60217645e-19 ** 2 / (4 * np.pi * 8.854187817e-12 * 1e-10)
STILL2, THRESHOLD, EPS_IN, EPS_OUT = 100.0, -4.0, 1.0, 80.0


def _orders(a, b, e):
    """Bond orders (1, 2, 3, else 7) of atoms [b, e) with every atom."""
    n = len(a["charge"])
    o = torch.full((e - b, n), 7, dtype=torch.int8, device=_device())
    for name, order in (("cov14", 3), ("cov13", 2), ("cov12", 1)):
        ptr, idx = a[name + "_ptr"], a[name + "_idx"]
        rows = np.repeat(np.arange(b, e), np.diff(ptr[b:e + 1]))
        o[torch.as_tensor(rows - b, device=_device()), torch.as_tensor(idx[ptr[b]:ptr[e]].astype(np.int64),
                                                                       device=_device())] = order
    return o


def _switch(r, rin, rc):
    """Energy switch S and dS/dr."""
    d, w = r - rin, (1.0 / (rc - rin)) ** 2
    s = 1.0 - w * d * d
    on = r >= rin
    return torch.where(on, s * s, torch.ones_like(r)), torch.where(on, -4.0 * w * d * s, torch.zeros_like(r))


def _force_switch(r, ri, rc):
    """Force-switched Coulomb: potential and force per unit charge product."""
    a = 1.0 / (rc ** 2 - ri ** 2) ** 3
    b, c, d = -(rc ** 6 - 3.0 * rc ** 4 * ri ** 2), 6.0 * rc ** 2 * ri ** 2, -(rc ** 2 + ri ** 2)
    f = lambda x: a * (b / x + c * x + d * x ** 3 + 0.4 * x ** 5)  # noqa: E731
    w = rc * rc - r * r
    on = r > ri
    return (torch.where(on, f(rc) - f(r), 1.0 / r - 1.0 / ri - (f(ri) - f(rc))),
            torch.where(on, -a * w * w * (rc * rc - 3 * ri * ri + 2 * r * r) / (r * r), -1.0 / (r * r)))


def _bonded(a, x):
    """Bonded forces, their energies and the bond virial (kcal/mol, A)."""
    t = lambda k, d=None: torch.as_tensor(np.asarray(a[k], dtype=d or np.float64), device=x.device)  # noqa: E731
    x = x.detach().clone().requires_grad_(True)
    k_J = 1.0 / KCAL
    i, j = t("bond_ij", np.int64).T
    lk = t("bond_lk")
    r = (x[i] - x[j]).norm(dim=1)
    bond = (lk[:, 1] * k_J * (r - lk[:, 0]) ** 2).sum()
    virial = (r * 2 * lk[:, 1] * k_J * (r - lk[:, 0])).sum()
    i, m, j = t("angle_iaj", np.int64).T
    kt = t("angle_kt")
    u, w = x[i] - x[m], x[j] - x[m]
    cs = (u * w).sum(1) / (u.norm(dim=1) * w.norm(dim=1))
    angle = (kt[:, 0] * k_J * (torch.acos(cs) - kt[:, 1]) ** 2).sum()
    tors = x.new_zeros(())
    for p in ("tors", "impr"):
        if not len(a[p + "_terms"]):
            continue
        q = t(p + "_idx", np.int64).reshape(-1, 4).T
        par, terms = t(p + "_par").reshape(-1, 12), t(p + "_terms", np.int64)
        va, vb, vc = x[q[0]] - x[q[1]], x[q[1]] - x[q[2]], x[q[2]] - x[q[3]]
        n1, n2 = torch.cross(va, vb, dim=1), torch.cross(vb, vc, dim=1)
        n3 = torch.cross(vb, n1, dim=1)
        phi = -torch.atan2((n3 * n2).sum(1) / n3.norm(dim=1), (n1 * n2).sum(1) / n1.norm(dim=1))
        for f in range(4):
            v, n, g = par[:, f], par[:, 4 + f], par[:, 8 + f]
            d = phi - g
            d = torch.where(d < -np.pi, d + 2 * np.pi, torch.where(d > np.pi, d - 2 * np.pi, d))
            e = torch.where(n > 0, 1.0 + torch.cos(n * phi + g), d * d)
            tors = tors + (torch.where(terms > f, v, torch.zeros_like(v)) * k_J * e).sum()
    (bond + angle + tors).backward()
    return -x.grad, {k: v.detach() for k, v in (("epot_bond", bond), ("epot_angle", angle), ("epot_torsion", tors),
                                                ("InternalVirial", virial))}


def _nonbonded(a, x, rc, mode):
    """Forces and energies of the non-bonded terms (kcal/mol, A); mode "gb"
    (GB + LJ + Coulomb), "energy" (the energies-only path) or "vacuum"."""
    dev, n, rin = x.device, len(x), rc - 3.0
    t = lambda k: torch.as_tensor(np.asarray(a[k], dtype=np.float64), device=dev)  # noqa: E731
    q, rad, eps = t("charge"), t("radius"), t("epsilon") / np.sqrt(KCAL)
    p4, p5, vdw14, elec14 = a["ff_params"][3], a["ff_params"][4], float(a["ff_params"][5]), float(a["ff_params"][6])
    chunks = [(b, min(n, b + 512)) for b in range(0, n, 512)]
    force = torch.zeros_like(x)
    out = {k: x.new_zeros(()) for k in ("epot_vdw", "epot_elec", "cross", "virial")}

    def geometry(b, e, reach2):
        d = x[b:e, None, :] - x[None, :, :]
        r2 = (d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2]
        near = r2 <= reach2
        near[torch.arange(e - b, device=dev), torch.arange(b, e, device=dev)] = False
        i, j = near.nonzero(as_tuple=True)
        return i + b, j, d[i, j], r2[i, j], _orders(a, b, e)[i, j]

    if mode != "vacuum":
        gbr, vj, total = t("gb_radius"), t("gb_vj"), t("gb_terms123").clone()
        still = []
        for b, e in chunks:
            i, j, d, r2, bo = geometry(b, e, STILL2)
            k = bo > 2
            i, j, d, r2 = i[k], j[k], d[k], r2[k]
            ratio = r2 / (gbr[i] + gbr[j]) ** 2
            th = ratio * p5 * np.pi
            far = ratio > 1.0 / p5
            s = 0.5 - 0.5 * torch.cos(th)
            ccf = torch.where(far, torch.ones_like(s), s * s)
            dccf = torch.where(far, torch.zeros_like(s), 2.0 * s * torch.sin(th) * th)
            total.index_add_(0, i, p4 * vj[j] * ccf / (r2 * r2))
            still.append((i, j, d, p4 * vj[j] * (4.0 * ccf - dccf) / r2 ** 3))
        born = -0.5 * ECONV / total
        premul = -0.5 * ECONV * (1.0 / EPS_IN - 1.0 / EPS_OUT)
        self_energy = premul * q * q / born
        deda = -self_energy / born
    for b, e in chunks:
        i, j, d, r2, bo = geometry(b, e, rc * rc)
        r = r2.sqrt()
        qq, nb, b14 = q[i] * q[j], bo > 2, bo == 3
        s, ds = _switch(r, rin, rc)
        coul = ECONV * (1.0 + (elec14 - 1.0) * b14.double()) * qq * nb
        radial = torch.zeros_like(r)
        if mode == "vacuum":
            pot, fr = _force_switch(r, rin, rc)
            ec, fe = coul * pot, coul * fr
        else:
            aa = born[i] * born[j]
            u = -0.25 * r2 / aa
            ec = coul / r
            if mode == "gb":
                on = u > THRESHOLD
                tg = torch.exp(u)
                g = (r2 + tg * aa).rsqrt()
                pol = torch.where(on, premul * qq * g, torch.zeros_like(g))
                fr = -pol * (r - 0.25 * r * tg) * g * g
                radial = 2.0 * (s * fr + ds * pol)
                deda.index_add_(0, i, -pol * tg * (1.0 - u) * g * g * s * born[j])
                out["cross"] += (pol * s).sum()
                ec = torch.where(on, ec / EPS_IN, ec / EPS_OUT)
            else:
                out["cross"] += (premul * qq * s * (r2 + torch.exp(u) * aa).rsqrt()).sum()
            fe = s * (-ec / r) + ds * ec
            ec = ec * s
        lj6 = ((rad[i] + rad[j]) / r) ** 6
        el = (1.0 + (vdw14 - 1.0) * b14.double()) * eps[i] * eps[j] * nb * (r < rc)
        ev, fv = 2.0 * el * (0.5 * lj6 * lj6 - lj6), -12.0 * el / r * (lj6 * lj6 - lj6)
        ev, fv = ev * s, s * fv + ds * ev
        force.index_add_(0, i, -((radial + fe + fv) / r)[:, None] * d)
        out["epot_vdw"] += 0.5 * ev.sum()
        out["epot_elec"] += 0.5 * ec.sum()
        out["virial"] += 0.5 * (r * (fe + fv)).sum()
    if mode == "vacuum":
        return force, {"epot_vdw": out["epot_vdw"], "epot_elec": out["epot_elec"], "InternalVirial": out["virial"]}
    out["self"] = self_energy.sum()
    if mode == "energy":
        return force, {"epot_vdw": out["epot_vdw"], "epot_elec": out["epot_elec"], "gb": out["cross"] + out["self"],
                       "InternalVirial": out["virial"]}
    weight = born * born / 166.0 * deda
    for i, j, d, g in still:
        f = (weight[i] * g)[:, None] * d
        force.index_add_(0, i, f).index_add_(0, j, -f)
    return force, {"epot_vdw": out["epot_vdw"], "epot_elec": out["epot_elec"], "epot_pol": out["cross"] + out["self"],
                   "epot_pol_cross": out["cross"], "epot_pol_self": out["self"]}


def _surface(a, x):
    """LCPO areas and, by differentiation, the forces of sigma * area (kcal/mol, A)."""
    use = torch.as_tensor(np.flatnonzero(a["lcpo_use"]), device=x.device)
    r = torch.as_tensor(np.asarray(a["lcpo_radius"], dtype=np.float64), device=x.device)[use]
    p = torch.as_tensor(np.asarray(a["lcpo_p"], dtype=np.float64).reshape(-1, 4), device=x.device)[use]
    y = x[use].detach().clone().requires_grad_(True)
    i, j = torch.nonzero(torch.cdist(y.detach(), y.detach(), compute_mode="donot_use_mm_for_euclid_dist") <
                         r[:, None] + r[None, :], as_tuple=True)
    i, j = i[i != j], j[i != j]
    d = (y[i] - y[j]).norm(dim=1)
    area = 2.0 * np.pi * r[i] * (r[i] - 0.5 * d - 0.5 * (r[i] ** 2 - r[j] ** 2) / d)
    n = len(use)
    overlap = torch.zeros(n, n, dtype=y.dtype, device=y.device).index_put((i, j), area)
    mask = (overlap.detach() != 0).double()
    inner = mask @ overlap.T  # [i, j]: sum of A_jk over the k that overlap both
    sasa = p[:, 0] * 4.0 * np.pi * r * r + p[:, 1] * overlap.sum(1) + p[:, 2] * (mask * inner).sum(1) + \
        p[:, 3] * (overlap * inner).sum(1)
    sasa = torch.where(sasa > 0, sasa, torch.zeros_like(sasa))
    energy = (ASP * sasa).sum()
    energy.backward()
    full, grad = torch.zeros(len(x), dtype=y.dtype, device=x.device), torch.zeros_like(x)
    full[use], grad[use] = sasa.detach(), y.grad
    return full, grad, energy.detach()


def _single(case, system, pos):
    """(forces in N, energies in J by name, sasa, SASAderiv) of one system."""
    a = _arrays(system)
    x = torch.as_tensor(pos, device=_device())
    mode = {"energy": "energy", "vacuum": "vacuum"}.get(case["kind"], "gb")
    force, ene = _bonded(a, x)
    f2, e2 = _nonbonded(a, x, case["cutoff"], mode)
    force = force + f2
    for k, v in e2.items():
        ene[k] = ene.get(k, 0.0) + v
    ene["epot"] = sum(ene[k] for k in ("epot_vdw", "epot_elec", "epot_bond", "epot_angle", "epot_torsion")) + \
        ene.get("epot_pol", 0.0) + ene.pop("gb", 0.0)
    sasa = deriv = None
    if case["kind"] == "surface":
        sasa, deriv, ene["epot_surf"] = _surface(a, x)
        force = force - deriv
        ene["epot"] = ene["epot"] + ene["epot_surf"]
        sasa, deriv = sasa.cpu().numpy(), -deriv.cpu().numpy()
    return force.cpu().numpy() * (KCAL / 1e-10), {k: float(v) * KCAL for k, v in ene.items()}, sasa, deriv


def _slots(ene):
    e = np.zeros(A.ENE_COUNT)
    for k, slot in pdgpu.Hamiltonian.FIELDS.items():
        e[slot] = ene.get(k, 0.0)
    return e


def exact(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] in ("forces", "energy", "vacuum", "surface"):
        f, ene, sasa, deriv = _single(case, case["system"], _displaced(case["system"], rng))
        if case["kind"] == "forces":
            return {"forces": f, "energies": _slots(ene)}
        out = {"forces": f, "energies": np.array([ene.get(k, 0.0) for k in FIELDS])}
        if case["kind"] == "surface":
            out.update(sasa=sasa, deriv=deriv)
        return out
    if case["kind"] == "serve":
        names = _members(case)
        pick = np.random.default_rng(case["jobs"]).integers(0, len(names), case["jobs"])
        got = [_single(case, names[k], _displaced(names[k], rng)) for k in pick]
        return {"forces": np.concatenate([f for f, *_ in got]), "energies": np.array([_slots(e) for _, e, *_ in got])}
    # the protocols' outputs follow the device's counter-based random numbers
    # or a chain of accepted steps: no closed form
    return None
