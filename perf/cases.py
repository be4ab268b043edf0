"""Performance cases of the solver and of the FDPS drop-in, through the public
entry points, over the range of sizes and options they are used at.

Kinds of case:

* ``steps``   a device-resident simulation (``Solver.step``) advanced a number
              of steps and read back, as a program does between two snapshots:
              dam breaks and periodic lattices, plain FP32 / FP32 tiled / half2,
              searching every step or with neighbour lists, one instance or an
              ensemble of uneven ones in one solver.
* ``probe``   one density pass and one force pass on a fixed state
              (``Solver.probe``), the force-kernel microbenchmark.
* ``device``  the walk pair sum on device-resident records
              (``wcsph_hydro_walks_noalloc``).
* ``fdps``    dispatch + retrieve of a multiwalk from host records, the hydro
              pair sum or the Shepard filter.

States come from the seed: positions jittered off the lattice, random
velocities and density fluctuations, as in a flow under way.
"""
import ctypes as C
import functools
import math

import numpy as np
import torch

from weaklycompressiblesph_b200 import _native as N
from weaklycompressiblesph_b200 import cases as setups
from weaklycompressiblesph_b200 import fdps
from weaklycompressiblesph_b200.sim import Solver

PRECISION = {"fp32": N.PREC_FP32, "tiled": N.PREC_TILED, "half2": N.PREC_HALF2}
NEIGHBOURS = 70          # in-support neighbours per particle at h = 1.3 dx, walls and surfaces included
PAIR_FLOPS, DENSITY_FLOPS = 60, 15
SHEPARD_INTERVAL = setups.Physics().shepard_interval
WALK_MARGIN = 0.15       # j-lists reach this many dx past the support: FDPS hands out supersets


def listed():
    return [
        # the solver with its default options, as small as the tests use it: launches and the read count
        {"name": "plain fp32 dam, 5k", "kind": "steps", "setup": "dam", "dx": 0.05, "precision": "fp32", "lists": 0,
         "steps": 25},
        # the small dam break of the reference's CPU runs (16,000 fluid particles), with neighbour lists
        {"name": "lists dam, 55k", "kind": "steps", "setup": "dam", "dx": 0.02, "precision": "tiled", "lists": 30,
         "steps": 25},
        # the headline workload: 1.02M fluid and 0.57M wall particles, FP32 neighbour lists, between two snapshots
        {"name": "lists dam, 1.6M", "kind": "steps", "setup": "dam", "dx": 0.005, "precision": "tiled", "lists": 30,
         "steps": 50},
        # the half-width record path at a middle size, dx not dividing the tank
        {"name": "half2 lists dam, 0.5M", "kind": "steps", "setup": "dam", "dx": 0.0079, "precision": "half2",
         "lists": 30, "steps": 50},
        # search every step: results that do not depend on the mix of instances (serving's library default)
        {"name": "search dam, 0.3M", "kind": "steps", "setup": "dam", "dx": 0.0097, "precision": "tiled", "lists": 0,
         "steps": 25},
        # periodic box with summation density every step; fast particles, so lists are rebuilt every few steps
        {"name": "lists lattice, 1M", "kind": "steps", "setup": "lattice", "side": 100, "precision": "tiled",
         "lists": 10, "steps": 10},
        # uneven dam breaks stepping together in half2, the ensemble workload
        {"name": "half2 ensemble of 8", "kind": "steps", "setup": "ensemble", "count": 8, "mix": 2024,
         "n_max": 1.0e5, "precision": "half2", "lists": 30, "steps": 25},
        # the force-kernel microbenchmark: one density and one force pass on the jittered periodic lattice
        {"name": "force probe lattice, 2M", "kind": "probe", "side": 127, "precision": "tiled", "density": 1},
        # walks of an application that owns all device memory: small and ragged, force.h's pair terms
        {"name": "device walks, 5k", "kind": "device", "dx": 0.05, "group": 50, "pair": "reference_cpu"},
        # the same at the FDPS group size, kernel.cu's pair terms (v_sig over the whole walk)
        {"name": "device walks, 0.3M", "kind": "device", "dx": 0.01, "group": 128, "pair": "reference_gpu"},
        # the FDPS drop-in from host records, as calcForceAllAndWriteBackMultiWalk drives it
        {"name": "fdps hydro, 0.16M", "kind": "fdps", "what": "hydro", "dx": 0.0125, "group": 128,
         "pair": "reference_gpu"},
        # the Shepard filter in the same shape
        {"name": "fdps filter, 0.16M", "kind": "fdps", "what": "filter", "dx": 0.0125, "group": 128,
         "pair": "reference_cpu"},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "probe", "device", "fdps"])
    if kind == "steps":
        c = {"kind": kind, "setup": rng.choice(["dam", "dam", "dam", "lattice", "ensemble"])}
        c["precision"] = rng.choice(["tiled", "tiled", "half2", "fp32"])
        c["lists"] = 0 if c["precision"] == "fp32" else rng.choice([0, 10, 30, 30])
        c["steps"] = rng.randint(5, 40)
        if c["setup"] == "dam":
            c["dx"] = round(_log_uniform(rng, 0.0055, 0.05), 5)
        elif c["setup"] == "lattice":
            c["side"] = int(_log_uniform(rng, 16, 110))
            c["steps"] = min(c["steps"], 10)
        else:
            c["count"], c["mix"] = rng.randint(2, 8), rng.randint(1, 10 ** 6)
            c["n_max"] = round(_log_uniform(rng, 2.0e4, 1.0e5))
        return c
    if kind == "probe":
        return {"kind": kind, "side": int(_log_uniform(rng, 16, 127)), "precision": rng.choice(["fp32", "tiled", "half2"]),
                "density": rng.randint(0, 2)}
    c = {"kind": kind, "dx": round(_log_uniform(rng, 0.011, 0.05), 5), "group": rng.randint(20, 128),
         "pair": rng.choice(["reference_gpu", "reference_cpu"])}
    if kind == "fdps":
        c["what"] = rng.choice(["hydro", "hydro", "filter"])
    return c


# ------------------------------------------------------------------ setups
@functools.lru_cache(maxsize=2)
def _dam(dx):
    return setups.dam_break(dx=dx)


@functools.lru_cache(maxsize=2)
def _ensemble(count, mix, n_max):
    return tuple(setups.ensemble_cases(count=count, seed=mix, n_min=1.0e4, n_max=n_max))


def _stirred(base, rng):
    """A dam break under way: fluid off its lattice, moving, compressed and stretched a little."""
    c = setups.Case(**{**base.__dict__})
    fluid = base.type == N.HYDRO
    c.pos = base.pos + np.where(fluid[:, None], rng.uniform(-0.05, 0.05, base.pos.shape) * base.dx, 0.0)
    c.vel = np.where(fluid[:, None], rng.normal(0.0, 0.3, base.vel.shape), 0.0)
    c.dens = base.dens * (1.0 + rng.uniform(-0.003, 0.003, base.n))
    return c


def _instances(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "probe" or case["setup"] == "lattice":
        return [setups.periodic_lattice(n_side=case["side"], dx=0.01, seed=seed)]
    if case["setup"] == "dam":
        return [_stirred(_dam(case["dx"]), rng)]
    return [_stirred(b, rng) for b in _ensemble(case["count"], case["mix"], case["n_max"])]


@functools.lru_cache(maxsize=2)
def _walks(dx, group):
    base = _dam(dx)
    return fdps.build_walks(base.pos, 2.0 * base.h + WALK_MARGIN * dx, group_size=group)


def _walk_case(case, seed):
    """Walks and FP64 records of a dam break under way."""
    c = _stirred(_dam(case["dx"]), np.random.default_rng(seed))
    w = _walks(case["dx"], case["group"])
    pres, snds = c.eos()
    epi, epj = fdps.walk_records(w, c.pos, c.vel, c.dens, pres, snds, c.h, c.mass, c.phys.nu, type_=c.type)
    if case.get("what") == "filter":
        fi, fj = np.zeros(len(epi), fdps.EPI_FILTER), np.zeros(len(epj), fdps.EPJ_FILTER)
        for f in fi.dtype.names:
            fi[f] = epi[f]
        for f in fj.dtype.names:
            fj[f] = epj[f]
        epi, epj = fi, fj
    return w, epi, epj


def _packed(w, epi, epj):
    """The device-resident FP32 records: positions relative to each walk's first i-particle."""
    origin = epi["pos"][w.i_off[:-1]]
    out = []
    for r, off in ((epi, w.i_off), (epj, w.j_off)):
        p = np.zeros((len(r), 3, 4), np.float32)
        p[:, 0, :3] = r["pos"] - np.repeat(origin, np.diff(off), axis=0)
        p[:, 0, 3] = r["smth"]
        p[:, 1, :3] = r["vel"]
        p[:, 1, 3] = r["dens"]
        p[:, 2, 0] = r["pres"] / r["dens"] ** 2
        p[:, 2, 1] = r["snds"]
        p[:, 2, 2] = r["visc"]
        if "mass" in r.dtype.names:
            p[:, 2, 3] = r["mass"]
        out.append(p)
    return out


# --------------------------------------------------------------- the calls
def prepare(case, seed):
    if case["kind"] in ("steps", "probe"):
        inst = _instances(case, seed)
        s = Solver(sum(c.n for c in inst) + 1024, precision=PRECISION[case["precision"]],
                   max_instances=len(inst) + 1, list_interval=case.get("lists", 0))
        return {"case": case, "solver": s, "slots": [s.add(c) for c in inst]}
    pair = fdps.pair_params(case["pair"], alpha=0.1)
    w, epi, epj = _walk_case(case, seed)
    n_i, n_j = np.diff(w.i_off).astype(np.int32), np.diff(w.j_off).astype(np.int32)
    st = {"case": case, "pair": pair, "n_walk": w.n_walk}
    if case["kind"] == "device":
        ri, rj = _packed(w, epi, epj)
        st.update({k: torch.from_numpy(v).cuda() for k, v in
                   (("n_i", n_i), ("n_j", n_j), ("epi", ri), ("epj", rj))})
        st["out"] = torch.empty((len(epi), 2, 4), dtype=torch.float32, device="cuda")
        return st
    fdps.configure(pair)
    out = np.zeros(len(epi), fdps.RESULT_FILTER if case["what"] == "filter" else fdps.RESULT_HYDRO)
    at = lambda a, off: (C.c_void_p * w.n_walk)(*(a.ctypes.data + off[:-1] * a.itemsize).tolist())  # noqa: E731
    st.update(epi=epi, epj=epj, out=out, n_i=n_i, n_j=n_j, p_i=at(epi, w.i_off), p_j=at(epj, w.j_off),
              p_o=at(out, w.i_off))
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "steps":
        st["solver"].step(case["steps"])
        return [st["solver"].read(k) for k in st["slots"]]
    if case["kind"] == "probe":
        return st["solver"].probe(st["slots"][0], density_pass=case["density"])
    if case["kind"] == "device":
        N.call("wcsph_hydro_walks_noalloc", st["n_walk"], C.c_void_p(st["n_i"].data_ptr()),
               C.c_void_p(st["n_j"].data_ptr()), C.c_void_p(st["epi"].data_ptr()), C.c_void_p(st["epj"].data_ptr()),
               C.c_void_p(st["out"].data_ptr()), C.byref(st["pair"]),
               C.c_void_p(torch.cuda.current_stream().cuda_stream))
        return {"acc_divv": st["out"][:, 0], "dt": st["out"][:, 1, 0]}
    what = case["what"]
    n_i, n_j = N.ptr(st["n_i"], C.c_int32), N.ptr(st["n_j"], C.c_int32)
    N.call(f"wcsph_{what}_dispatch", 0, st["n_walk"], st["p_i"], n_i, st["p_j"], n_j)
    N.call(f"wcsph_{what}_retrieve", 0, st["n_walk"], n_i, st["p_o"])
    return {f: st["out"][f] for f in st["out"].dtype.names}


def _dam_count(dx, column=(0.4, 0.4, 0.8), tank=(1.6, 0.4, 1.0), layers=3):
    c, t = [round(v / dx) for v in column], [round(v / dx) for v in tank]
    box = (t[0] + 2 * layers) * (t[1] + 2 * layers) * (t[2] + layers)
    return c[0] * c[1] * c[2] + box - t[0] * t[1] * t[2]


def work(case):
    """State (position, velocity, density, acceleration, div v) or records in once, results out once; the
    arithmetic of every in-support pair."""
    if case["kind"] in ("steps", "probe"):
        if case["kind"] == "probe" or case["setup"] == "lattice":
            n = case["side"] ** 3
        elif case["setup"] == "dam":
            n = _dam_count(case["dx"])
        else:
            n = sum(c.n for c in _ensemble(case["count"], case["mix"], case["n_max"]))
        pairs = NEIGHBOURS * n
        if case["kind"] == "probe":
            return {"bytes": n * (28 + 28), "flops": pairs * (PAIR_FLOPS + (DENSITY_FLOPS if case["density"] else 0))}
        every = 1 if case["setup"] == "lattice" else 1.0 / SHEPARD_INTERVAL
        return {"bytes": n * (44 + 48), "flops": case["steps"] * pairs * (PAIR_FLOPS + every * DENSITY_FLOPS)}
    n, w = _dam_count(case["dx"]), _walks(case["dx"], case["group"])
    n_j = len(w.j_idx)
    if case["kind"] == "device":
        return {"bytes": 48 * (n + n_j) + 32 * n, "flops": NEIGHBOURS * n * PAIR_FLOPS}
    if case["what"] == "filter":
        return {"bytes": 32 * n + 40 * n_j + 8 * n, "flops": NEIGHBOURS * n * DENSITY_FLOPS}
    return {"bytes": 96 * n + 112 * n_j + 40 * n, "flops": NEIGHBOURS * n * PAIR_FLOPS}


# ------------------------------------------------- the same in 64 bits, torch
class _Exact:
    """One instance in FP64 from the FP32 state the solver is given."""

    def __init__(self, c):
        t = lambda a: torch.from_numpy(np.asarray(a, np.float32)).cuda().double()  # noqa: E731
        self.p, self.x, self.v, self.rho = c.phys, t(c.pos), t(c.vel), t(c.dens)
        self.h, self.m, self.H = c.h, c.mass, 2.0 * c.h
        self.fluid = torch.from_numpy(np.asarray(c.type)).cuda() == N.HYDRO
        self.box = torch.tensor(np.array(c.hi) - np.array(c.lo), device="cuda") if c.periodic else None
        self.nbr = None
        self.x_ref = None

    def _image(self, d):
        return d if self.box is None else d - self.box * torch.round(d / self.box)

    def _neighbours(self):
        """nbr[i]: the particles within 2.6 h of i, padded with i; built again once something moved 0.25 h."""
        if self.x_ref is not None and float((self.x - self.x_ref).norm(dim=1).max()) < 0.25 * self.h:
            return
        self.x_ref = x = self.x.clone()
        R, dev = 2.6 * self.h, x.device
        if self.box is None:
            lo = x.min(0).values
            nc = ((x.max(0).values - lo) / R).floor().long() + 1
            edge = torch.full((3,), R, device=dev, dtype=torch.float64)
            y = x
        else:
            lo = torch.zeros(3, device=dev, dtype=torch.float64)
            nc = (self.box / R).floor().long().clamp(min=1)
            edge = self.box / nc
            y = x - self.box * torch.floor(x / self.box)
        cell = torch.minimum(((y - lo) / edge).long(), nc - 1)
        key = (cell[:, 2] * nc[1] + cell[:, 1]) * nc[0] + cell[:, 0]
        ks, order = key.sort()
        count = torch.bincount(ks, minlength=int(nc.prod()))
        start = count.cumsum(0) - count
        n, occ = len(x), int(count.max())
        off = torch.tensor([[a, b, c] for c in (-1, 0, 1) for b in (-1, 0, 1) for a in (-1, 0, 1)], device=dev)
        if self.box is not None:  # few cells an axis: visit each neighbour cell once
            off = torch.unique(off % nc, dim=0)
        slot = torch.arange(occ, device=dev)
        rows, step = [], max(1, 60_000_000 // (len(off) * occ))
        for a in range(0, n, step):
            i = torch.arange(a, min(n, a + step), device=dev)
            q = cell[i][:, None, :] + off
            if self.box is None:
                ok = ((q >= 0) & (q < nc)).all(2)
            else:
                q, ok = q % nc, torch.ones(q.shape[:2], dtype=torch.bool, device=dev)
            k = torch.where(ok, (q[..., 2] * nc[1] + q[..., 1]) * nc[0] + q[..., 0], 0)
            there = ok[..., None] & (slot < count[k][..., None])
            j = order[torch.where(there, start[k][..., None] + slot, 0)].reshape(len(i), -1)
            d = self._image(x[i][:, None] - x[j])
            hit = there.reshape(len(i), -1) & ((d * d).sum(2) < R * R) & (j != i[:, None])
            width = int(hit.sum(1).max())
            first = torch.sort(hit.int(), dim=1, descending=True, stable=True).indices[:, :width]
            rows.append(torch.where(hit.gather(1, first), j.gather(1, first), i[:, None]).int())
        width = max(r.shape[1] for r in rows)
        self.nbr = torch.empty((n, width), dtype=torch.int32, device=dev)
        a = 0
        for r in rows:
            self.nbr[a:a + len(r), :r.shape[1]] = r
            self.nbr[a:a + len(r), r.shape[1]:] = torch.arange(a, a + len(r), device=dev, dtype=torch.int32)[:, None]
            a += len(r)

    def _chunks(self):
        self._neighbours()
        step = max(1, 30_000_000 // self.nbr.shape[1])
        for a in range(0, len(self.x), step):
            j = self.nbr[a:a + step]
            i = slice(a, a + len(j))
            d = [x[i, None] - x[j] for x in self.x.unbind(1)]
            if self.box is not None:
                d = [e - b * torch.round(e / b) for e, b in zip(d, self.box.tolist())]
            r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
            yield i, j, d, r2, (r2 > 0) & (r2 < self.H ** 2)

    def density(self, shepard):
        out = torch.empty_like(self.rho)
        for i, j, _, r2, inside in self._chunks():
            s = r2.sqrt() / self.H
            w = torch.where(inside, (1 - s).clamp(min=0) ** 3 - 4 * (0.5 - s).clamp(min=0) ** 3, 0.0)
            total = 0.5 + w.sum(1)
            if shepard:
                out[i] = total / (0.5 / self.rho[i] + (w / self.rho[j]).sum(1))
            else:
                out[i] = self.m * 16 / (math.pi * self.H ** 3) * total
        return out

    def force(self, v, rho):
        """Hydro acceleration, div v and each particle's dt."""
        p = self.p
        X = rho / p.rho0
        po = (p.B * (X ** p.gamma - 1)).clamp(min=0) / rho ** 2
        c = (p.B * p.gamma / p.rho0 * X ** (p.gamma - 1)).clamp(min=1e-16).sqrt()
        acc, divv, vsig = torch.empty_like(self.x), torch.empty_like(rho), torch.empty_like(rho)
        K = 16 / (math.pi * self.H ** 4)
        for i, j, d, r2, inside in self._chunks():
            r = r2.sqrt()
            s = r / self.H
            g = torch.where(inside, (12 * (0.5 - s).clamp(min=0) ** 2 - 3 * (1 - s).clamp(min=0) ** 2) * K /
                            r.clamp(min=1e-300), 0.0)
            dv = [u[i, None] - u[j] for u in v.unbind(1)]
            drdv = d[0] * dv[0] + d[1] * dv[1] + d[2] * dv[2]
            den = r2 + p.eps * self.h ** 2
            mu = torch.where(inside & (drdv < 0), self.h * drdv / den, 0.0)
            rs = rho[i, None] + rho[j]
            av = (p.beta * mu - p.alpha * 0.5 * (c[i, None] + c[j])) * mu * 2 / rs
            f = -(po[i, None] + po[j] + av) * g
            visc = 4 * p.nu * g * r2 / rs / den
            for k in range(3):
                acc[i, k] = self.m * (visc * dv[k] + f * d[k]).sum(1)
            divv[i] = -self.m * (g * drdv).sum(1) / rho[i]
            vsig[i] = (-mu).max(1).values
        return acc, divv, p.c_cfl * self.h / (c + vsig)

    def _pass(self, v):
        acc, divv, dt = self.force(v, self.rho)
        acc[:, 2] -= self.p.g
        self.rho = self.rho.clamp(min=self.p.rho_floor)
        limit = torch.minimum(dt, 0.25 * (self.h / acc.norm(dim=1)).sqrt())
        nu = 0.125 * self.h ** 2 / self.p.nu
        self.acc, self.divv, self.dt = acc, divv, min(float(limit[self.fluid].min()), nu)

    def steps(self, k):
        summation = self.p.density_mode == N.DENSITY_SUMMATION
        if summation:
            self.rho = self.density(False)
        before = self.rho
        self._pass(self.v)
        if not summation:
            self.rho = before
            self.rho = self.density(True).clamp(min=self.p.rho_floor)
        moving = self.fluid[:, None]
        for step in range(k):
            dt = self.dt
            self.rho = self.rho - self.rho * dt * self.divv
            half = self.v + 0.5 * dt * self.acc
            self.x = torch.where(moving, self.x + dt * half, self.x)
            v = torch.where(moving, self.v + dt * self.acc, self.v)
            if summation or step % SHEPARD_INTERVAL == 0:
                self.rho = self.density(not summation)
            self._pass(v)
            self.v = torch.where(moving, half + 0.5 * dt * self.acc, self.v)
        return {"pos": None if self.box is not None else self.x, "vel": self.v, "dens": self.rho, "acc": self.acc,
                "div_v": self.divv, "alive": None}


def _exact_walks(case, seed):
    w, epi, epj = _walk_case(case, seed)
    pair = fdps.pair_params(case["pair"], alpha=0.1)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda().double()  # noqa: E731
    if case["kind"] == "device":
        (xi, vi, ci), (xj, vj, cj) = ([t(p[:, k]) for k in range(3)] for p in _packed(w, epi, epj))
    elif case["what"] == "filter":
        xi, xj = t(np.c_[epi["pos"], epi["smth"]]), t(epj["pos"])
        mj, rj = t(epj["mass"]), t(epj["dens"])
    else:
        rec = lambda r, m: (t(np.c_[r["pos"], r["smth"]]), t(np.c_[r["vel"], r["dens"]]),  # noqa: E731
                            t(np.c_[r["pres"] / r["dens"] ** 2, r["snds"], r["visc"], m]))
        (xi, vi, ci), (xj, vj, cj) = rec(epi, np.zeros(len(epi))), rec(epj, epj["mass"])
    n = len(epi)
    acc = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    dt = torch.empty(n, dtype=torch.float64, device="cuda")
    grad = lambda r, h: torch.where(  # noqa: E731
        r < 2 * h, (12 * (0.5 - r / (2 * h)).clamp(min=0) ** 2 - 3 * (1 - r / (2 * h)).clamp(min=0) ** 2) *
        16 / (math.pi * (2 * h) ** 4) / r.clamp(min=1e-300), 0.0)
    for k in range(w.n_walk):
        i, j = slice(int(w.i_off[k]), int(w.i_off[k + 1])), slice(int(w.j_off[k]), int(w.j_off[k + 1]))
        d = xi[i, None, :3] - xj[None, j, :3]
        r2 = (d * d).sum(2)
        r, hi = r2.sqrt(), xi[i, 3:4]
        if case.get("what") == "filter":
            s = r / (2 * hi)
            W = (1 - s).clamp(min=0) ** 3 - 4 * (0.5 - s).clamp(min=0) ** 3
            dt[i] = (W * mj[j]).sum(1) / (W * (mj[j] / rj[j])).sum(1)
            continue
        hj = xj[None, j, 3]
        dv = vi[i, None, :3] - vj[None, j, :3]
        drdv = (d * dv).sum(2)
        den = r2 + pair.eps * hi * hj
        mu = torch.where((drdv < 0) & (r2 > 0), 0.5 * (hi + hj) * drdv / den, 0.0)
        g = 0.5 * (grad(r, hi) + grad(r, hj)) if pair.grad_mode else grad(r, 0.5 * (hi + hj))
        g = torch.where(r2 > 0, g, 0.0)
        rho = vi[i, 3:4] + vj[None, j, 3]
        av = (-pair.alpha * 0.5 * (ci[i, 1:2] + cj[None, j, 1]) * mu + pair.beta * mu * mu) * 2 / rho
        f = (ci[i, 0:1] + cj[None, j, 0] + av) * g
        visc = 2 * (ci[i, 2:3] + cj[None, j, 2]) * g * r2 / rho / den
        m = cj[None, j, 3]
        acc[i, :3] = (m[..., None] * (visc[..., None] * dv - f[..., None] * d)).sum(1)
        acc[i, 3] = -(m * g * drdv).sum(1) / vi[i, 3]
        vsig = ((-mu) if pair.vsig_mode else mu).max(1).values.clamp(min=0)
        dt[i] = pair.c_cfl * hi[:, 0] / (ci[i, 1] + vsig)
    if case["kind"] == "device":
        return {"acc_divv": acc, "dt": dt}
    if case["what"] == "filter":
        return {"dens": dt}
    return {"acc": acc[:, :3], "dt": dt, "div_v": acc[:, 3]}


def exact(case, seed):
    if case["kind"] in ("device", "fdps"):
        return _exact_walks(case, seed)
    inst = _instances(case, seed)
    if case["kind"] == "steps":
        return [_Exact(c).steps(case["steps"]) for c in inst]
    e = _Exact(inst[0])
    # adding the instance runs its initial summation density (the lattice's density mode)
    e.rho = e.density(False).float().double()
    if case["density"]:
        e.rho = e.density(case["density"] == 2)
    acc, divv, dt = e.force(e.v, e.rho)
    return {"acc": acc, "div_v": divv, "dt": dt, "dens": e.rho, "nbr": None}
