"""The work that a user has this library do, as cases to time.

Every case goes through the public Python entry points (``plan_gb300.Finder`` and
``plan_gb300.Server``) the way a program calls them: snapshots are .lis records in page-locked
host memory, groups and query positions are host arrays, results come back to the host.

kinds
  find       one snapshot through build_tree + find_planetesimals: the clump catalogue, and the density
             that the finder gave each particle.
  serve      several snapshots of mixed sizes through the serving loop, submitted at once.
  neighbours build_tree of a snapshot, then the k nearest tree points of some of its particles.
  knn        the neighbour queries alone, on a tree that the program has built before.
  dvs        build_tree with density_vs_scale, then the densest sphere of every radius.
  energies   kinetic and potential energies of a batch of particle groups (boundness).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import plan_gb300 as pg


# ---------------------------------------------------------------- the cases
def _find(n: int, mix: str, nx: int, knn: int = 32, hop: int = 16, time: float = 0.0) -> dict:
    return {"kind": "find", "n": n, "mix": mix, "nx": nx, "knn": knn, "hop": hop, "time": time}


def listed() -> list[dict]:
    return [
        # the test-sized snapshot: what a user runs first, and what a parameter scan repeats; latency and launches count
        dict(_find(20000, "spheres", 32), name="find 20k"),
        # few particles on a fine grid: fewer than four particles per horizontal cell takes the spline density
        dict(_find(50000, "spheres", 128), name="find 50k spline"),
        # the plain method's own configuration: 262,144 particles, 16 spheres
        dict(_find(262144, "spheres", 128), name="find 262k"),
        # an odd-sized snapshot in mid-run, sheared, with more neighbours than the default
        dict(_find(100003, "spheres", 64, knn=48, hop=24, time=0.37), name="find 100k sheared knn48"),
        # the benchmark's mixture (background, sheets, clumps): a production snapshot
        dict(_find(524288, "filaments", 128), name="find 524k filaments"),
        # an early snapshot of a run: filaments, nothing collapsed yet; the particles are the work, not the clumps
        dict(_find(1500000, "early", 128), name="find 1.5m early"),
        # a run's output directory handed to the serving loop: mixed sizes, several in flight
        {"name": "serve 6 mixed", "kind": "serve", "n_lo": 65536, "n_hi": 262144, "requests": 6, "workers": 3},
        # the benchmark's snapshot size: its tree, then the neighbours of a few hundred particles of interest
        {"name": "tree 16.7m + neighbours", "kind": "neighbours", "n": 16777216, "mix": "filaments", "nx": 128, "queries": 500, "k": 32},
        # neighbour lists of many particles of an ordinary snapshot
        {"name": "knn 100k queries", "kind": "knn", "n": 1000000, "mix": "filaments", "nx": 128, "queries": 100000, "k": 32},
        # the density-vs-scale analysis on a grid of 32 cells a side
        {"name": "dvs 150k nx32", "kind": "dvs", "n": 150000, "mix": "spheres", "nx": 32, "time": 0.37},
        # the boundness of the few candidate groups of one small snapshot
        {"name": "energies 16 small", "kind": "energies", "groups": 16, "n_lo": 32, "n_hi": 1000},
        # the batched boundness benchmark: thousands of groups of tens to thousands of particles
        {"name": "energies 5000 mixed", "kind": "energies", "groups": 5000, "n_lo": 32, "n_hi": 20000},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng) -> dict:
    """One more case of the same ranges."""
    kind = rng.choice(["find", "find", "find", "serve", "neighbours", "knn", "dvs", "energies", "energies"])
    if kind == "find":
        mix = rng.choice(["spheres", "filaments", "early"])
        n = _log(rng, 5000, {"spheres": 262144, "filaments": 400000, "early": 1500000}[mix]) | 1
        nx = rng.choice([32, 64, 128])
        knn, hop = rng.choice([(32, 16), (32, 16), (24, 12), (48, 24), (64, 32)])
        return _find(n, mix, nx, knn, hop, rng.choice([0.0, 0.0, round(rng.uniform(0.1, 1.5), 3)]))
    if kind == "serve":
        lo = _log(rng, 16000, 65536)
        return {"kind": "serve", "n_lo": lo, "n_hi": _log(rng, 65536, 262144), "requests": rng.randint(2, 6), "workers": rng.randint(2, 4)}
    if kind == "neighbours":
        return {"kind": "neighbours", "n": _log(rng, 100000, 16000000) | 1, "mix": rng.choice(["spheres", "filaments", "early"]), "nx": 128,
                "queries": _log(rng, 1, 5000), "k": rng.choice([8, 16, 31, 32, 64])}
    if kind == "knn":
        return {"kind": "knn", "n": _log(rng, 20000, 1000000) | 1, "mix": rng.choice(["spheres", "filaments", "early"]), "nx": 128,
                "queries": _log(rng, 1, 100000), "k": rng.choice([1, 8, 16, 32, 33, 64, 100])}
    if kind == "dvs":
        return {"kind": "dvs", "n": _log(rng, 5000, 150000) | 1, "mix": rng.choice(["spheres", "filaments"]), "nx": rng.choice([8, 16, 24, 32]),
                "time": rng.choice([0.0, round(rng.uniform(0.05, 1.5), 3)])}
    n_hi = _log(rng, 100, 100000)
    # the number of groups keeps the pairs below the largest listed batch's
    return {"kind": "energies", "groups": max(1, min(5000, _log(rng, 1, max(2.0, 2e11 / (n_hi * n_hi))))), "n_lo": rng.choice([1, 32, 77]), "n_hi": n_hi}


# ---------------------------------------------------------------- inputs
class _Snapshot:
    """A snapshot whose records are already in page-locked host memory (pg.Snapshot without the file)."""

    def __init__(self, n: int, mix: str, nx: int, time: float, seed: int):
        spec = pg.SynthSpec()
        L = pg.lib()
        L.plan_synth_default_spec(1 if mix == "spheres" else 2, n, seed, C.byref(spec))
        spec.nx = nx
        spec.time = time
        if mix == "early":
            spec.n_clumps = 0
        self.four_pi_G = L.plan_synth_four_pi_G_for_mean(C.byref(spec), nx, nx)
        spec.G = self.four_pi_G / (4 * math.pi)
        self.rec = torch.empty(n * 44, dtype=torch.uint8, pin_memory=torch.cuda.is_available())
        info = pg.SynthInfo()
        rc = L.plan_synth_records(C.byref(spec), C.c_void_p(self.rec.data_ptr()), C.byref(info))
        if rc:
            raise pg.PlanError(rc, "snapshot generator")
        v = pg.LisView()
        for i in range(12):
            v.coor_lim[i] = float(np.float32((-0.1, 0.1)[i % 2]))
        v.ntypes = 1
        v.type_info[0] = 1.0
        v.time = time
        v.nblocks = 1
        self._ptr, self._cnt = (C.c_void_p * 1)(self.rec.data_ptr()), (C.c_uint64 * 1)(n)
        v.records = C.cast(self._ptr, C.POINTER(C.c_void_p))
        v.counts = C.cast(self._cnt, C.POINTER(C.c_uint64))
        self.view = v

    def positions(self) -> np.ndarray:
        return self.rec.numpy().reshape(-1, 44)[:, :12].copy().view(np.float32).astype(np.float64)


def _params(snap: _Snapshot, nx: int, knn: int = 32, hop: int = 16) -> pg.Params:
    """What pg.params reads from a parameter file with these values."""
    p = pg.params()
    p.box_resolution[:] = (nx, nx, nx)
    p.solid_to_gas_ratio = 0.02
    p.four_pi_G = snap.four_pi_G
    p.knn, p.hop, p.fixed_hop = knn, hop, 1
    return p


def _groups(case: dict, seed: int):
    """Plummer groups (scale 1e-3) with particles of 0.5 to 1.5 times the mean mass, sizes log-uniform."""
    rng = np.random.default_rng(seed)
    sizes = np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"] + 0.999), case["groups"])).astype(np.int64)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    n = int(off[-1])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    gen = torch.Generator(dev).manual_seed(seed)
    r = 1e-3 / torch.sqrt((1e-6 + 0.99 * torch.rand(n, generator=gen, device=dev)) ** (-2.0 / 3.0) - 1.0)
    d = torch.randn(n, 3, generator=gen, device=dev)
    centre = torch.from_numpy(rng.uniform(-0.09, 0.09, (len(sizes), 3)).astype(np.float32)).to(dev)
    pos = torch.repeat_interleave(centre, torch.from_numpy(sizes).to(dev), dim=0) + r[:, None] * d / d.norm(dim=1, keepdim=True)
    vel = 1e-3 * torch.randn(n, 3, generator=gen, device=dev)
    mass = 4.0106053e-08 * (0.5 + torch.rand(n, generator=gen, device=dev))
    return pos.cpu().numpy(), vel.cpu().numpy(), mass.cpu().numpy(), off


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "energies":
        p = pg.params()
        pg.lib().plan_params_derive(C.byref(p))
        return {"kind": kind, "groups": _groups(case, seed), "params": p, "finder": pg.Finder(0)}
    if kind == "serve":
        rng = np.random.default_rng(seed)
        jobs = []
        for i in range(case["requests"]):
            n = int(np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]))))
            snap = _Snapshot(n, "filaments", 128, 0.0, seed * 1000 + i)
            jobs.append((snap, _params(snap, 128)))
        return {"kind": kind, "jobs": jobs, "server": pg.Server(0, case["workers"], 0)}
    snap = _Snapshot(case["n"], case["mix"], case["nx"], case.get("time", 0.0), seed)
    p = _params(snap, case["nx"], case.get("knn", 32), case.get("hop", 16))
    state = {"kind": kind, "snap": snap, "params": p, "finder": pg.Finder(0)}
    if kind == "dvs":
        p.density_vs_scale = 1
    if kind in ("neighbours", "knn"):
        pick = np.random.default_rng(seed).integers(0, case["n"], case["queries"])
        state["queries"] = np.ascontiguousarray(snap.positions()[pick])
        state["k"] = case["k"]
    if kind == "knn":
        state["finder"].build_tree(snap, p)
    return state


# ---------------------------------------------------------------- one pass
_ROWS = 512  # of the table that a program keeps per snapshot; there are far fewer clumps


def _catalogue(cat: pg.Catalogue) -> dict:
    """The catalogue as a table: its first `count` rows, the others zero."""
    ids, val = np.zeros((_ROWS, 2), np.int64), np.zeros((_ROWS, 11))
    n = 0
    for n, c in enumerate(cat.clumps(), 1):
        ids[n - 1] = c["peak_id"], c["npar"]
        val[n - 1] = (c["total_mass"], c["hill_radius"], *c["com"], *c["vel_com"], *c["J"])
    cat.close()
    return {"count": n, "ids": ids, "values": val}


def _densities(finder: pg.Finder, n: int) -> np.ndarray:
    """Each particle's density; the tree points of ghosts and of particles folded into another are left out."""
    orig, dens = finder.stage(pg.PLAN_ARR_ORIG_ID), finder.stage(pg.PLAN_ARR_DENSITY)
    own = orig < n
    out = np.zeros(n)
    out[orig[own]] = dens[own]
    return out


def run(state: dict):
    kind = state["kind"]
    if kind == "find":
        out = _catalogue(state["finder"].find_clumps(state["snap"], state["params"]))
        out["density"] = _densities(state["finder"], int(state["snap"].view.counts[0]))
        return out
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(snap, p) for snap, p in state["jobs"]]
        return [_catalogue(srv.poll(i, wait=True)[0]) for i in ids]
    if kind == "neighbours":
        state["finder"].build_tree(state["snap"], state["params"])
        return state["finder"].knn(state["queries"], state["k"])
    if kind == "knn":
        return state["finder"].knn(state["queries"], state["k"])
    if kind == "dvs":
        state["finder"].build_tree(state["snap"], state["params"])
        return state["finder"].density_vs_scale(state["params"], state["snap"].view.time)
    ek, ep, zeros = state["finder"].group_energies(*state["groups"], state["params"])
    return ek, ep, zeros


# ---------------------------------------------------------------- the work a pass cannot do without
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "find":
        # the records in, the densities and the catalogue out, a distance to each neighbour of both searches
        return {"bytes": 52 * case["n"] + 1000, "flops": 8 * case["n"] * (case["knn"] + case["hop"])}
    if kind == "serve":
        n = case["requests"] * math.sqrt(case["n_lo"] * case["n_hi"])
        return {"bytes": int(44 * n), "flops": int(8 * n * 48)}
    if kind == "neighbours":
        return {"bytes": 44 * case["n"] + case["queries"] * (24 + 12 * case["k"]), "flops": 8 * case["queries"] * case["k"]}
    if kind == "knn":
        return {"bytes": case["queries"] * (24 + 12 * case["k"]), "flops": 8 * case["queries"] * case["k"]}
    if kind == "dvs":
        # every cell centre and sub-centre needs at least one distance
        return {"bytes": 44 * case["n"] + 200, "flops": 8 * 39 * case["nx"] ** 3}
    lo, hi = case["n_lo"], case["n_hi"] + 0.999
    s = math.log(hi / lo)
    mean, mean2 = (hi - lo) / s, (hi * hi - lo * lo) / (2 * s)
    # a pair: three differences, a squared distance, its reciprocal root, the mass, the sum
    return {"bytes": int(case["groups"] * (28 * mean + 24)), "flops": int(case["groups"] * (mean2 - mean) / 2 * 11)}


# ---------------------------------------------------------------- the same in 64 bits
def exact(case: dict, seed: int):
    """Energies by direct sums in FP64, radii of density_vs_scale. Catalogues and neighbour lists follow the
    reference's own search rules and orders; they have no plain form and are whole numbers or compared bit by bit."""
    if case["kind"] == "dvs":
        cell = 2 * float(np.float32(0.1)) / case["nx"]
        nlev = round(math.log10(case["nx"]) / math.log10(2.0)) + 1
        return np.array([cell / 2 * 2.0 ** i for i in range(nlev)]), None
    if case["kind"] != "energies":
        return None
    pos, vel, mass, off = _groups(case, seed)
    p = pg.params()
    pg.lib().plan_params_derive(C.byref(p))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, v, m = (torch.from_numpy(a).to(dev).double() for a in (pos, vel, mass))
    ek, ep = np.zeros(case["groups"]), np.zeros(case["groups"])
    dek, dep = [], []
    for g in range(case["groups"]):
        b, e = int(off[g]), int(off[g + 1])
        xg, vg, mg = x[b:e], v[b:e], m[b:e]
        M = mg.sum()
        xc, vc = (mg[:, None] * xg).sum(0) / M, (mg[:, None] * vg).sum(0) / M
        dv = vc - vg
        dv[:, 1] -= p.q * p.Omega * (xc[0] - xg[:, 0])
        dek.append(0.5 * (mg * (dv * dv).sum(1)).sum())
        pot = torch.zeros((), dtype=torch.float64, device=dev)
        for i in range(0, e - b, 4096):  # rows [i, i + 4096) against the columns from i on
            d = torch.cdist(xg[i:i + 4096], xg[i:], compute_mode="donot_use_mm_for_euclid_dist").reciprocal_()
            d.masked_fill_(torch.isinf(d), 0.0)
            r = d.shape[0]
            pot += mg[i:i + r] @ (d @ mg[i:]) - 0.5 * (mg[i:i + r] @ (d[:, :r] @ mg[i:i + r]))
        dep.append(pot)
    if dek:
        ek, ep = torch.stack(dek).cpu().numpy(), -p.grav_constant * torch.stack(dep).cpu().numpy()
    return ek, ep, None
