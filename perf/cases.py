"""The work that users of this library have it do, as cases that can be timed.

Each case is one call (or the two or three that belong together) through the
public entry points, on seeded face-centred-cubic copper near the temperatures
the tests and the benchmark use:

  force      comdgb_force on an attached simflat_t: the potential's force pointer
  steps      comdgb_sim_steps on a device-resident handle, then the state by id
  dropin     comdgb_nTimeSteps on an attached simflat_t, state copied both ways
  batch      comdgb_sim_graph_steps over replicas of several sizes, then each state
  loss_grad  comdgb_sim_force_loss_grad: one force-matching gradient
  traj_grad  comdgb_sim_traj_energy_grad: the gradient through a trajectory
  analysis   virial tensor, per-atom stress and centrosymmetry of one frame

The mixed-precision path computes its pair terms in FP32, so what it yields is
handed on in FP32 here; positions, which it integrates in FP64, stay FP64.
"""
import ctypes as C
import math
import os
import struct

import numpy as np
import torch

import comd_gb300 as cg

LATTICE, MASS = 3.615, 63.55                    # copper: A, amu
LJ = {"sigma": 2.315, "epsilon": 0.167 / 27.211386245988, "cutoff": 2.5 * 2.315}
AMU, KB, TIME = 1822.83, 3.166811563e-6, 0.529 / 2.418e-17
DT = 1e-15
POTS = {"lj": cg.POT_LJ, "table": cg.POT_EAM_TABLE, "cheby": cg.POT_EAM_CHEBY}
SLOTS = 64
GPU = "cuda"


def _case(name, kind, pot, prec, nx, ny, nz, bf=1.0, stretch=1.0, temp=300.0, disp=0.05, **more):
    return dict(name=name, kind=kind, pot=pot, prec=prec, nx=nx, ny=ny, nz=nz, bf=bf,
                stretch=stretch, temp=temp, disp=disp, periodic=True, **more)


def listed():
    return [
        # the smallest call: the force pointer of a host program on 4,000 LJ atoms
        _case("lj_force_4k", "force", "lj", "fp64", 10, 10, 10),
        # the default options but for open boundaries, on a ragged slab
        dict(_case("table_force_26k_open", "force", "table", "fp64", 17, 19, 20), periodic=False),
        # the 256,000-atom FP64 table run of the configurations
        _case("table_steps_256k_fp64", "steps", "table", "fp64", 40, 40, 40, temp=600.0, n=20),
        # the Chebyshev potential in FP64, as a reference run of a mixed one
        _case("cheby_steps_108k_fp64", "steps", "cheby", "fp64", 30, 30, 30, bf=1.2, n=10),
        # a host program's own loop: nTimeSteps(10) between its energy prints
        _case("cheby_dropin_1m_mixed", "dropin", "cheby", "mixed", 64, 64, 64, bf=1.5,
              stretch=1.05, n=10),
        # a small system run for long: bound by launches and latency
        _case("cheby_steps_4k_mixed", "steps", "cheby", "mixed", 10, 10, 10, bf=1.2, n=100),
        # the benchmark's lattice
        _case("cheby_steps_4m_mixed", "steps", "cheby", "mixed", 100, 100, 100, bf=1.5,
              stretch=1.05, disp=0.0, n=50),
        # the table potential in mixed precision, edges that divide nothing
        _case("table_steps_282k_mixed", "steps", "table", "mixed", 41, 40, 43, bf=1.2, temp=600.0,
              n=50),
        # replicas of edge 8 to 24 cells at 100 to 1200 K, advanced together
        _case("batch_24_mixed", "batch", "cheby", "mixed", 8, 24, 24, bf=1.2, disp=0.0, n=20,
              replicas=24),
        # one configuration of a potential fit
        _case("loss_grad_256k", "loss_grad", "cheby", "fp64", 40, 40, 40),
        # the backward pass through a short trajectory
        _case("traj_grad_4k", "traj_grad", "cheby", "fp64", 9, 10, 11, n=20, every=10),
        # what is written beside a frame
        _case("analysis_256k", "analysis", "cheby", "fp64", 40, 40, 40),
    ]


def _edges(rng, lo, hi, most):
    """three edges of about the same size, log-uniform, odd ones among them"""
    while True:
        e = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        n = [max(lo, round(e * rng.uniform(0.85, 1.18))) for _ in range(3)]
        if 4 * n[0] * n[1] * n[2] <= most:
            return n


def draw(rng):
    kind = rng.choice(["force", "force", "steps", "steps", "steps", "dropin", "batch", "loss_grad",
                       "traj_grad", "analysis"])
    pot, prec, bf = rng.choice(["table", "cheby"]), rng.choice(["fp64", "mixed"]), rng.choice([1.0, 1.2])
    temp, more, periodic = round(rng.uniform(100.0, 900.0), 1), {}, True
    if kind == "force":
        pot = rng.choice(["lj", "table", "cheby"])
        periodic = rng.random() < 0.75
        edges = _edges(rng, 7, 50, 500_000)
    elif kind == "steps":
        edges = _edges(rng, 6, 92, 3_000_000) if prec == "mixed" else _edges(rng, 6, 42, 280_000)
        more["n"] = rng.randint(10, 50) if prec == "mixed" else rng.randint(5, 15)
    elif kind == "dropin":
        edges = _edges(rng, 6, 64, 1_000_000) if prec == "mixed" else _edges(rng, 6, 30, 100_000)
        more["n"] = rng.randint(1, 10)
    elif kind == "batch":
        lo = rng.randint(6, 10)
        edges = [lo, rng.randint(lo + 2, 24), 24]
        prec = "mixed" if rng.random() < 0.7 else "fp64"
        more = {"n": rng.randint(5, 20 if prec == "mixed" else 8), "replicas": rng.randint(3, 24)}
    elif kind == "traj_grad":
        pot, prec, edges = "cheby", "fp64", _edges(rng, 6, 12, 6_000)
        more = {"n": rng.randint(5, 20), "every": rng.randint(3, 12)}
    else:
        pot, prec, edges = "cheby", "fp64", _edges(rng, 7, 40, 256_000)
        if kind == "analysis":
            pot = rng.choice(["table", "cheby"])
    c = _case("", kind, pot, prec, *edges, bf=bf, temp=temp,
              disp=round(rng.uniform(0.01, 0.08), 3), **more)
    del c["name"]
    c["periodic"] = periodic
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _replicas(case):
    """one case per replica of a batch: edges and temperatures spread over the range"""
    lo, hi, m = case["nx"], case["ny"], case["replicas"]
    out = []
    for r in range(m):
        # (a stride coprime to the count spreads sizes over the order)
        e = [lo + (7 * r + 5 * q + r * r) % (hi - lo + 1) for q in range(3)]
        out.append(dict(case, nx=e[0], ny=e[1], nz=e[2], temp=100.0 + 1100.0 * ((5 * r) % m) / m))
    return out


def _inputs(case, seed):
    """world positions and momenta by id, and the box: FP64 on the GPU"""
    g = torch.Generator(device=GPU).manual_seed(int(seed))
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    k, j, i = torch.meshgrid(*(torch.arange(2 * n, device=GPU) for n in (nz, ny, nx)), indexing="ij")
    at = torch.stack([i, j, k], -1).reshape(-1, 3)
    at = at[at.sum(1) % 2 == 1].double()
    unit = torch.tensor([LATTICE * case["stretch"], LATTICE, LATTICE], dtype=torch.float64, device=GPU)
    x = (at * 0.5 + 0.25) * unit
    box = unit * torch.tensor([nx, ny, nz], dtype=torch.float64, device=GPU)
    if case["disp"]:
        x = x + case["disp"] * torch.randn(x.shape, dtype=torch.float64, device=GPU, generator=g)
    p = math.sqrt(MASS * AMU * KB * case["temp"]) * torch.randn(
        x.shape, dtype=torch.float64, device=GPU, generator=g)
    p = p - p.mean(0)  # no drift of the whole lattice
    return x, p, box


def _cutoff(case):
    return LJ["cutoff"] if case["pot"] == "lj" else _tables()["phi"]["xn"]


def _layout(case, x, box):
    """slot of every atom, in id order within its box, and the boxes' corners and counts"""
    rc = _cutoff(case)
    b = box.cpu().numpy()
    strain = [case["stretch"], 1.0, 1.0]
    nbx = [int(math.floor(b[m] / (rc * case["bf"] * strain[m]))) for m in range(3)]
    size = torch.tensor([b[m] / nbx[m] for m in range(3)], dtype=torch.float64, device=GPU)
    top = torch.tensor(nbx, device=GPU) - 1
    ix = torch.minimum(torch.floor(x / size).long().clamp(min=0), top)
    nb = nbx[0] * nbx[1] * nbx[2]
    where = ix[:, 0] + nbx[0] * (ix[:, 1] + nbx[1] * ix[:, 2])
    order = torch.argsort(where, stable=True)
    count = torch.bincount(where, minlength=nb)
    start = torch.cumsum(count, 0) - count
    rank = torch.empty_like(where)
    rank[order] = torch.arange(len(where), device=GPU) - start[where[order]]
    return where * SLOTS + rank, x - ix * size, count, nbx


class Host:
    """A host simflat_t with the atoms of one case; frees what it owns."""

    def __init__(self, case, seed):
        self.L = cg.load()
        self.attached = False
        if case["pot"] == "lj":
            self.pot = cg.lj_potential(LJ["sigma"], LJ["epsilon"], LJ["cutoff"], MASS)
        else:
            self.pot = cg.eam_potential("cu")
        self.s = cg.fcc(case["nx"], case["ny"], case["nz"], LATTICE, case["stretch"], case["bf"],
                        self.pot)
        s = self.s.contents
        x, p, box = _inputs(case, seed)
        slot, r, count, nbx = _layout(case, x, box)
        assert list(s.nbx) == nbx and s.ntot == len(x) and int(count.max()) < SLOTS
        n = s.nboxes * SLOTS
        self.view("natoms")[:] = count.int().cpu().numpy()
        for name, v in (("r", r), ("p", p)):
            full = torch.zeros((n, 3), dtype=torch.float64, device=GPU)
            full[slot] = v
            torch.from_numpy(self.view(name)).copy_(full)
        ids = torch.zeros(n, dtype=torch.int32, device=GPU)
        ids[slot] = torch.arange(len(x), dtype=torch.int32, device=GPU)
        torch.from_numpy(self.view("id")).copy_(ids)
        self.view("mass")[:] = MASS
        self.view("iType")[:] = 1

    def view(self, name):
        """a slot array as numpy sees it; it keeps this simulation alive"""
        s = self.s.contents
        n = s.nboxes * (1 if name == "natoms" else SLOTS)
        wide = {"r": 3, "p": 3, "f": 4}.get(name, 1)
        t = C.c_int if name in ("natoms", "id", "iType") else C.c_double
        a = (t * (n * wide)).from_address(C.cast(getattr(s, name), C.c_void_p).value)
        a.owner = self
        a = np.ctypeslib.as_array(a)
        return a.reshape(n, wide) if wide > 1 else a

    def attach(self, o):
        cg.lib.check(self.L.comdgb_attach(self.s, C.byref(o)))
        self.attached = True

    def __del__(self):
        if getattr(self, "s", None):
            if self.attached:
                self.L.comdgb_detach(self.s)
            cg.free_host(self.s)
            self.s = None


def _opts(case):
    return cg.opts(POTS[case["pot"]], cg.PREC_MIXED if case["prec"] == "mixed" else cg.PREC_FP64,
                   periodic=case["periodic"])


def _target(case, seed, n):
    g = torch.Generator(device=GPU).manual_seed(int(seed) + 77)
    return 0.02 * torch.randn((n, 3), dtype=torch.float64, device=GPU, generator=g)


def prepare(case, seed):
    st = {"case": case}
    kind = case["kind"]
    if kind in ("force", "dropin"):
        st["host"] = Host(case, seed)
        st["host"].attach(_opts(case))
    elif kind == "batch":
        hosts = [Host(c, seed * 101 + r) for r, c in enumerate(_replicas(case))]
        st["pot"] = hosts[0].pot
        st["sim"] = cg.Batch([h.s for h in hosts], _opts(case))
    else:
        host = Host(case, seed)
        st["pot"] = host.pot
        st["sim"] = cg.DeviceSim(host.s, _opts(case))
        if kind == "loss_grad":
            st["target"] = _target(case, seed, host.s.contents.ntot).cpu().numpy()
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _narrow(mixed):
    """results of the mixed path in the precision they carry"""
    if not mixed:
        return lambda v: v
    return lambda v: torch.from_numpy(v).float() if isinstance(v, np.ndarray) else np.float32(v)


def run(state):
    case = state["case"]
    kind, n = case["kind"], case.get("n", 0)
    low = _narrow(case["prec"] == "mixed")
    if kind == "force":
        h = state["host"]
        cg.lib.check(h.L.comdgb_force(h.s))
        s = h.s.contents
        out = {"e": low(s.e), "stress": low(s.stress), "f": low(h.view("f"))}
        if case["pot"] != "lj":
            out.update(rho=low(h.view("rho")), fi=low(h.view("fi")))
        return out
    if kind == "dropin":
        h = state["host"]
        e = h.L.comdgb_nTimeSteps(n, h.s, DT)
        if not math.isfinite(e):
            raise RuntimeError(cg.lib.last_error())
        out = {"e": low(e), "stress": low(h.s.contents.stress), "natoms": h.view("natoms"),
               "id": h.view("id"), "r": h.view("r")}
        for name in ("p", "f", "rho", "fi"):
            out[name] = low(h.view(name))
        return out
    sim = state["sim"]
    if kind == "steps":
        e, stress = sim.steps(n, DT)
        return dict({"e": low(e), "stress": low(stress)}, **_atoms(sim.gather(), low))
    if kind == "batch":
        sim.graph_steps(n, DT)
        e, stress = sim.energies()
        g = np.concatenate([sim.gather(r) for r in range(sim.n)])
        return dict({"e": low(e), "stress": low(stress)}, **_atoms(g, low))
    if kind == "loss_grad":
        loss, grad = sim.force_loss_grad(state["target"])
        return {"loss": loss, "grad": grad}
    if kind == "traj_grad":
        j, grad = sim.traj_energy_grad(n, DT, case["every"])
        return dict({"j": j, "grad": grad}, **_atoms(sim.gather(), low))
    w, k, volume = sim.virial()
    centro, lo, hi = sim.centrosymmetry()
    return {"w": w, "k": k, "volume": volume, "atom": sim.atom_stress(), "centro": centro,
            "lo": lo, "hi": hi}


def _atoms(g, low):
    return {"x": g[:, :3], "p": low(g[:, 3:])}


def work(case):
    cases = _replicas(case) if case["kind"] == "batch" else [case]
    atoms = sum(4 * c["nx"] * c["ny"] * c["nz"] for c in cases)
    pairs = atoms * (39 if case["pot"] == "lj" else 21)  # unique ones within the cutoff
    per_pair, per_atom = (30, 10) if case["pot"] == "lj" else (60, 40)
    force = pairs * per_pair + atoms * per_atom
    kind, n = case["kind"], case.get("n", 0)
    if kind == "force":  # positions in; force and energy, and for EAM rho and F' out
        return {"bytes": atoms * (24 + 32 + (0 if case["pot"] == "lj" else 16)), "flops": force}
    if kind in ("steps", "dropin", "batch"):  # a step reads and writes positions and momenta
        return {"bytes": atoms * (96 * n + 96 + (64 if kind == "dropin" else 0)),
                "flops": force * (n + 1) + atoms * 18 * n}
    if kind == "loss_grad":  # 32 terms of three weighted sums over the pairs
        return {"bytes": atoms * 48, "flops": force + pairs * 32 * 8}
    if kind == "traj_grad":  # forward, and per step back a gradient and a Hessian product
        return {"bytes": atoms * 96 * 2 * n, "flops": n * (2 * force + pairs * 32 * 8 + pairs * 100)}
    # virial terms, and twelve nearest of the neighbours with their best pairing
    return {"bytes": atoms * (48 + 48 + 8), "flops": force + pairs * 40 + atoms * (42 * 9 + 66 * 8)}


# ---------------------------------------------------------------------------
# the same results in 64 bits by torch
# ---------------------------------------------------------------------------
def _tables():
    """the copper tables: guard cells and the raised x0 as the format defines them"""
    if not _tables.read:
        for name in ("phi", "rho", "f"):
            with open(os.path.join(cg.POT_DIR, "cu." + name), "rb") as fp:
                raw = fp.read()
            e = ">" if struct.unpack("<i", raw[:4])[0] > 4096 else "<"
            n, x0, xn, inv, lo, hi = struct.unpack(e + "idddii", raw[4:40])
            v = np.frombuffer(raw, e + "f8", n, 48).astype(np.float64)
            end = v[-1] if hi else 0.0
            v = np.concatenate([[v[0] if lo else 0.0], v, [end, end]])
            _tables.read[name] = {"n": n, "x0": x0 + (xn - x0) / n, "xn": xn, "inv": inv, "v": v}
    return _tables.read


_tables.read = {}


def _interpolate(t, r):
    """value and derivative of a table"""
    v = torch.from_numpy(t["v"]).to(r.device)
    u = (r.clamp(t["x0"], t["xn"]) - t["x0"]) * t["inv"]
    i = torch.floor(u).long().clamp(0, t["n"] - 1)
    u = u - i
    a, b, c, d = v[i], v[i + 1], v[i + 2], v[i + 3]
    g0, g1 = c - a, d - b
    val = b + 0.5 * u * (u * (c + a - 2.0 * b) + g0)
    return val, torch.where(i > 0, 0.5 * (g0 + u * (g1 - g0)) * t["inv"], torch.zeros_like(u))


def _fit(t, m=32):
    """the coefficients of a table's Chebyshev series on [x0, xn]"""
    k = np.arange(m)
    y = np.cos(np.pi * (k + 0.5) / m)
    r = y * 0.5 * (t["xn"] - t["x0"]) + 0.5 * (t["xn"] + t["x0"])
    f = _interpolate(t, torch.from_numpy(r))[0].numpy()
    f = np.where(f > 1e10, 0.0, f)
    return 2.0 / m * np.cos(np.pi * np.outer(k, k + 0.5) / m) @ f


def _slope(m=32):
    """coefficients of the derivative (in y) of a series from its own"""
    d = np.zeros((m, m))
    d[m - 2, m - 1] = 2.0 * (m - 1)
    for j in range(m - 2, 0, -1):
        d[j - 1] = d[j + 1]
        d[j - 1, j] += 2.0 * j
    return torch.from_numpy(d).to(GPU)


class Model:
    """Energy, forces and the rest of one potential over a list of pairs."""

    def __init__(self, pot):
        self.pot = pot
        if pot == "lj":
            self.rc = LJ["cutoff"]
            return
        t = _tables()
        self.rc = t["phi"]["xn"]
        if pot == "cheby":
            self.c = torch.from_numpy(np.stack([_fit(t[q]) for q in ("phi", "rho", "f")])).to(GPU)
            self.ends = [(t[q]["x0"], t[q]["xn"]) for q in ("phi", "rho", "f")]
            self.slope = _slope()

    def _series(self, c, q, x):
        a, b = self.ends[q]
        y = (2.0 * x.clamp(min=a) - a - b) / (b - a)
        d, dd = torch.zeros_like(y), torch.zeros_like(y)
        for j in range(len(c) - 1, 0, -1):
            d, dd = 2.0 * y * d - dd + c[j], d
        return y * d - dd + 0.5 * c[0]

    def function(self, q, x):
        """value and derivative of phi (0), rho (1) or F (2)"""
        if self.pot == "table":
            return _interpolate(_tables()[("phi", "rho", "f")[q]], x)
        a, b = self.ends[q]
        return (self._series(self.c[q], q, x),
                self._series((self.slope @ self.c[q]) * (2.0 / (b - a)), q, x))

    def terms(self, x, box, pairs, periodic):
        i, j = pairs
        d = x[i] - x[j]
        if periodic:
            d = d - box * torch.round(d.detach() / box)
        r2 = (d * d).sum(1)
        near = r2.detach() <= self.rc * self.rc
        return i[near], j[near], d[near], r2[near]

    def __call__(self, x, box, pairs, periodic=True):
        i, j, d, r2 = self.terms(x, box, pairs, periodic)
        n = len(x)
        both = lambda v: torch.zeros(n, dtype=v.dtype, device=GPU).index_add(0, i, v).index_add(0, j, v)  # noqa: E731
        if self.pot == "lj":
            s6 = LJ["sigma"] ** 6
            r6 = 1.0 / (r2 * r2 * r2)
            e = both(0.5 * r6 * (s6 * r6 - 1.0))
            w = 4.0 * LJ["epsilon"] * s6 * r6 / r2 * (12.0 * s6 * r6 - 6.0)
            total, out = 4.0 * LJ["epsilon"] * s6 * e.sum(), {}
        else:
            r = torch.sqrt(r2)
            (phi, dphi), (rho, drho) = self.function(0, r), self.function(1, r)
            dens = both(rho)
            emb, fi = self.function(2, dens)
            e = 0.5 * both(phi) + emb
            part = (fi[i] + fi[j]) * drho / r
            w = dphi / r + part
            total = e.sum()
            out = {"rho": dens, "fi": fi, "stress": 2.0 * (part * d[:, 0] ** 2).sum() / box.prod()}
        v = w[:, None] * d
        f = torch.zeros_like(x).index_add(0, i, v).index_add(0, j, -v)
        return dict(out, total=total, e=e, f=f, w=w, d=d, i=i, j=j)


def _pairs(x, box, rc, periodic=True):
    """unique pairs within rc (at least three cells of that width an edge)"""
    b = box.cpu().numpy()
    m = [max(3 if periodic else 1, int(b[q] // rc)) for q in range(3)]
    size = box / torch.tensor(m, dtype=torch.float64, device=GPU)
    y = x.detach()
    if periodic:
        y = torch.remainder(y, box)
    ix = torch.minimum(torch.floor(y / size).long().clamp(min=0), torch.tensor(m, device=GPU) - 1)
    cell = ix[:, 0] + m[0] * (ix[:, 1] + m[1] * ix[:, 2])
    nc = m[0] * m[1] * m[2]
    order = torch.argsort(cell, stable=True)
    count = torch.bincount(cell, minlength=nc)
    start = torch.cumsum(count, 0) - count
    wide = int(count.max())
    table = torch.full((nc, wide), -1, dtype=torch.long, device=GPU)
    table[cell[order], torch.arange(len(x), device=GPU) - start[cell[order]]] = order
    c = torch.arange(nc, device=GPU)
    at = [c % m[0], (c // m[0]) % m[1], c // (m[0] * m[1])]
    found = []
    for o in range(27):
        o = (o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1)
        if (o[2], o[1], o[0]) < (0, 0, 0):
            continue
        to = [at[q] + o[q] for q in range(3)]
        ok = torch.ones(nc, dtype=torch.bool, device=GPU)
        for q in range(3):
            if periodic:
                to[q] = to[q] % m[q]
            else:
                ok &= (to[q] >= 0) & (to[q] < m[q])
        src = c[ok]
        dst = (to[0] + m[0] * (to[1] + m[1] * to[2]))[ok]
        for part in range(0, len(src), 1 << 17):
            p, q = table[src[part:part + (1 << 17)]], table[dst[part:part + (1 << 17)]]
            d = y[p.clamp(min=0)][:, :, None] - y[q.clamp(min=0)][:, None]
            if periodic:
                d = d - box * torch.round(d / box)
            hit = ((d * d).sum(-1) <= rc * rc) & (p >= 0)[:, :, None] & (q >= 0)[:, None]
            if o == (0, 0, 0):
                hit &= p[:, :, None] < q[:, None]
            a, u, v = torch.nonzero(hit, as_tuple=True)
            found.append((p[a, u], q[a, v]))
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _verlet(model, x, p, box, n):
    """n steps and the force call that ends them"""
    h, m = DT * TIME, AMU * MASS
    for t in range(n + 1):
        if t % 20 == 0:
            pairs = _pairs(x, box, model.rc + 1.0)
        if t < n:
            x = x + 0.5 * h / m * p
            p = p - h * model(x, box, pairs)["f"]
            x = x + 0.5 * h / m * p
    return x, p, model(x, box, pairs)


def _centro(x, box, pairs):
    """least sum of |r_a + r_b|^2 over the pairings of the twelve nearest"""
    i, j = pairs
    d = x[j] - x[i]
    d = d - box * torch.round(d / box)
    i, d = torch.cat([i, j]), torch.cat([d, -d])
    r2 = (d * d).sum(1)
    order = torch.argsort(r2)
    order = order[torch.argsort(i[order], stable=True)]
    n = len(x)
    count = torch.bincount(i, minlength=n)
    first = torch.cumsum(count, 0) - count
    v = d[order[first[:, None] + torch.arange(12, device=GPU)]]  # [n, 12, 3]
    best = {0: torch.zeros(n, dtype=torch.float64, device=GPU)}
    for _ in range(6):  # subsets reached by pairing the lowest free one
        more = {}
        for used, val in best.items():
            a = next(q for q in range(12) if not used >> q & 1)
            for b in range(a + 1, 12):
                if not used >> b & 1:
                    s = val + ((v[:, a] + v[:, b]) ** 2).sum(1)
                    k = used | 1 << a | 1 << b
                    more[k] = s if k not in more else torch.minimum(more[k], s)
        best = more
    return best[4095]


def _by_slot(case, x, box, v):
    slot, _, count, _ = _layout(case, x, box)
    out = torch.zeros((len(count) * SLOTS,) + v.shape[1:], dtype=torch.float64, device=GPU)
    out[slot] = v
    return out


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    atoms = 4 * case["nx"] * case["ny"] * case["nz"]
    if kind in ("steps", "dropin") and atoms * n > 50_000_000:
        return None
    if kind == "batch":
        outs = [_exact(c, seed * 101 + r) for r, c in enumerate(_replicas(case))]
        return {"e": torch.stack([o["e"] for o in outs]),
                "stress": torch.stack([o["stress"] for o in outs]),
                "x": torch.cat([o["x"] for o in outs]), "p": torch.cat([o["p"] for o in outs])}
    return _exact(case, seed)


def _exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    x, p, box = _inputs(case, seed)
    model = Model(case["pot"])
    if kind == "force":
        o = model(x, box, _pairs(x, box, model.rc, case["periodic"]), case["periodic"])
        out = {"e": o["total"], "stress": o.get("stress"),
               "f": _by_slot(case, x, box, torch.cat([o["f"], o["e"][:, None]], 1))}
        for name in ("rho", "fi"):
            if name in o:
                out[name] = _by_slot(case, x, box, o[name])
        return out
    if kind in ("steps", "batch", "dropin"):
        y, q, o = _verlet(model, x, p, box, n)
        out = {"e": o["total"], "stress": o["stress"]}
        if kind != "dropin":  # (a drop-in call leaves its results by slot)
            out.update(x=torch.remainder(y, box), p=q)
        return out
    if kind == "loss_grad":
        model.c.requires_grad_(True)
        o = model(x, box, _pairs(x, box, model.rc))
        loss = ((o["f"] - _target(case, seed, len(x))) ** 2).sum()
        (grad,) = torch.autograd.grad(loss, model.c)
        return {"loss": loss.detach(), "grad": grad.reshape(-1)}
    if kind == "traj_grad":
        model.c.requires_grad_(True)
        y, q, o = _verlet(model, x, p, box, n)
        (grad,) = torch.autograd.grad(o["total"], model.c)
        return {"j": o["total"].detach(), "grad": grad.reshape(-1),
                "x": torch.remainder(y.detach(), box), "p": q.detach()}
    pairs = _pairs(x, box, model.rc)
    o = model(x, box, pairs)
    m = AMU * MASS
    voigt = ((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))
    k = torch.stack([p[:, a] * p[:, b] / m for a, b in voigt], 1)
    w = torch.stack([-0.5 * o["w"] * o["d"][:, a] * o["d"][:, b] for a, b in voigt], 1)
    w = torch.zeros_like(k).index_add(0, o["i"], w).index_add(0, o["j"], w)
    c = _centro(x, box, pairs)
    return {"w": w.sum(0), "k": k.sum(0), "volume": box.prod(),
            "atom": _by_slot(case, x, box, -(k + w)), "centro": _by_slot(case, x, box, c),
            "lo": c.min(), "hi": c.max()}
