"""Performance cases of the framework: the runs a user of it makes, through
its Python API (md_gpu_gb300.MDSystem), over the sizes of its own
configurations and tests.

Kinds (the value of a case's "kind"):

  argon     LJ argon, reaction-field kernel, velocity Verlet NVE (the
            framework's configuration "argon" is 4000 atoms; its tests go down
            to a few hundred)
  nvt       molten-salt NaCl, LJ + Wolf, Berendsen leapfrog (configuration
            "nacl64k" from its stored melt; smaller and ragged sizes as its
            replicas and tests have)
  host      the same system end to end from pinned host buffers (run_host):
            upload, list, energies, steps, download
  water     flexible water with bonds, angles and Nose-Hoover (configuration
            "water": 98304 atoms; its tests use a few thousand)
  pme       NaCl with Ewald electrostatics by particle-mesh Ewald
  npt       NaCl at constant pressure (Berendsen barostat)
  replicas  a batch of uneven NaCl replicas, velocity Verlet NVE (the
            benchmark's batch workload: 256 to 8192 ions each)
  point     energies and forces of configurations given one after the other
            (set_positions, compute_forces with energies, forces, energies)
  fp64      the FP64 mode of the force kernels, velocity Verlet NVE
  adjoint   loss and parameter gradients of a batch's trajectory

Positions, velocities and forces of FP32-mode runs come back as float32, the
precision of the forces that made them; the FP64 mode's come back as float64.
Positions after steps are given next to where they started (the run's own
periodic wrap taken off), as a user who follows displacements has them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import md_gpu_gb300 as md
from md_gpu_gb300 import synth

RGAS = 8.314e-3             # kJ/mol/K
QFAC = float(np.float32(1389.35427611722))     # kJ/mol A / e^2, as the force kernels hold it
BAR = 16605.3907            # bar per kJ/mol/A^3
A_S = [float(np.float32(a)) for a in (0.254829592, -0.284496736, 1.421413741, -1.453152027, 1.061405429)]
P_S = float(np.float32(0.3275911))


def listed():
    return [
        # the smallest runs: launch and synchronisation latency count
        {"name": "argon-500", "kind": "argon", "ncell": 5, "steps": 100, "energy_every": 0},
        # configuration "argon" at its size, energies every 50 steps
        {"name": "argon-4000", "kind": "argon", "ncell": 10, "steps": 100, "energy_every": 50},
        # a small, ragged molten-salt box, the reference's default loop
        {"name": "nvt-982", "kind": "nvt", "natom": 982, "steps": 100, "energy_every": 0, "tuned": False},
        # flexible water at test size: bonds, angles, exclusions, thermostat
        {"name": "water-5184", "kind": "water", "nside": 12, "steps": 20},
        # configuration "water" at its size
        {"name": "water-98304", "kind": "water", "nside": 32, "steps": 8},
        # the headline system from its stored melt, tuned as a production run is
        {"name": "nvt-64000", "kind": "nvt", "natom": 64000, "steps": 48, "energy_every": 0, "tuned": True},
        # the headline system end to end, untuned
        {"name": "host-64000", "kind": "host", "natom": 64000, "steps": 32},
        # long-range electrostatics on the headline system
        {"name": "pme-64000", "kind": "pme", "natom": 64000, "grid": 112, "steps": 16},
        # constant pressure, a few thousand ions
        {"name": "npt-7986", "kind": "npt", "natom": 7986, "steps": 32},
        # many uneven replicas advanced together (the largest work)
        {"name": "replicas-128", "kind": "replicas", "nrep": 128, "nmax": 8192, "steps": 48},
        # reference-precision run
        {"name": "fp64-4082", "kind": "fp64", "natom": 4082, "steps": 8},
        # gradients of a trajectory, as in parameter fitting
        {"name": "adjoint-16x1000", "kind": "adjoint", "nrep": 16, "natom": 1000, "steps": 20, "checkpoint": 10},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _ragged(rng, lo, hi):
    """An even ion count from lo to hi that leaves at most 4% of the sites of
    an even-sided lattice vacant (nacl_replica's lattice, no compressed start)."""
    sides = [m for m in range(8, 42, 2) if lo <= m ** 3 <= hi]
    t = _log(rng, lo, hi)
    m = min(sides, key=lambda s: abs(math.log(s ** 3 / t)))
    return m ** 3 - 2 * rng.randint(0, int(0.02 * m ** 3))


def draw(rng):
    kind = rng.choice(["argon", "argon", "nvt", "nvt", "host", "water", "pme", "npt", "replicas", "point", "fp64",
                       "adjoint"])
    if kind == "argon":
        return {"kind": kind, "ncell": rng.randint(4, 20), "steps": rng.randint(20, 128),
                "energy_every": rng.choice([0, 0, 10, 50])}
    if kind == "nvt":
        return {"kind": kind, "natom": _ragged(rng, 512, 64000), "steps": rng.randint(16, 48),
                "energy_every": rng.choice([0, 0, 10]), "tuned": rng.random() < 0.3}
    if kind == "host":
        return {"kind": kind, "natom": _ragged(rng, 512, 64000), "steps": rng.randint(8, 32)}
    if kind == "water":
        return {"kind": kind, "nside": rng.randint(8, 30), "steps": rng.randint(8, 20)}
    if kind == "pme":
        n = _ragged(rng, 1000, 64000)
        L = synth.nacl_replica(n).box[0]
        return {"kind": kind, "natom": n, "grid": 8 * math.ceil(L / rng.uniform(0.9, 1.2) / 8), "steps": rng.randint(8, 16)}
    if kind == "npt":
        return {"kind": kind, "natom": _ragged(rng, 1728, 32768), "steps": rng.randint(8, 40)}
    if kind == "replicas":
        return {"kind": kind, "nrep": int(_log(rng, 8, 128)), "nmax": rng.choice([1728, 4096, 8192]),
                "steps": rng.randint(16, 48)}
    if kind == "point":
        return {"kind": kind, "natom": _ragged(rng, 512, 64000)}
    if kind == "fp64":
        return {"kind": kind, "natom": _ragged(rng, 512, 8000), "steps": rng.randint(4, 16)}
    return {"kind": kind, "nrep": rng.randint(2, 16), "natom": _ragged(rng, 512, 1728), "steps": rng.randint(8, 20),
            "checkpoint": rng.choice([5, 10])}


# ---- systems: keyword arguments of MDSystem.from_arrays, from the seed alone ----

def _velocities(rng, type_mass, itype, temp):
    m = np.asarray(type_mass, np.float64)[itype]
    v = rng.standard_normal((len(itype), 3)) * np.sqrt(RGAS * temp / m)[:, None]
    return v - (v * m[:, None]).sum(0) / m.sum()


def _nacl(natom, seed, **kw):
    """NaCl of natom ions: the stored melt (64000), shifted as a whole and with
    new velocities, else a seeded lattice."""
    if natom != 64000:
        return synth.to_arrays(synth.nacl_replica(natom, seed=seed, nmaxlist=416, **kw))
    rng = np.random.default_rng(seed)
    a = synth.to_arrays(synth.nacl_melt64k())
    L = np.asarray(a["box"], np.float64)
    x = a["pos"].astype(np.float64) + rng.uniform(0.0, 1.0, 3) * L
    x -= L * np.floor(x / L + 0.5)
    a["pos"] = np.clip(x.astype(np.float32), -0.5 * a["box"], 0.5 * a["box"])
    a["vel"] = _velocities(rng, a["type_mass"], a["itype"], 1200.0).astype(np.float32)
    a.update(integrator=md.MD_VV if kw.get("integrator") == "vv" else md.MD_LEAPFROG,
             enstype={"nve": 0, "nvt": 1, "npt": 2}[kw.get("ensemble", "nvt")])
    return a


def _water(nside, seed):
    s = synth.water_grid(nside=nside, seed=seed)
    b, a = s.bonds.copy(), s.angles.copy()
    flat = dict(s.inp)
    s.bonds, s.angles = s.bonds[:0], s.angles[:0]
    kw = synth.to_arrays(s)
    b[:, 0:] -= 1
    a[:, 0:] -= 1
    kw.update(bonds=b, angles=a, nmaxlist=int(flat["skin"][1]),
              bnd1=[2.0 * k for k, _ in s.bond_types], bnd2=[r for _, r in s.bond_types],
              ang1=[2.0 * k for k, _ in s.angle_types], ang2=[math.radians(t) for _, t in s.angle_types])
    return kw


def _replica_sizes(case):
    rng = np.random.default_rng(case["nrep"])
    sides = [m for m in range(8, 22, 2) if m ** 3 <= case["nmax"]]
    out = []
    for _ in range(case["nrep"]):
        m = int(rng.choice(sides))
        out.append(m ** 3 - 2 * int(rng.integers(0, int(0.02 * m ** 3) + 1)))
    return out


def _systems(case, seed):
    """The systems of a case as from_arrays dicts (one, but for batches)."""
    k = case["kind"]
    if k == "argon":
        return [synth.to_arrays(synth.argon_fcc(ncell=case["ncell"], seed=seed, integrator="vv"))]
    if k in ("nvt", "host"):
        return [_nacl(case["natom"], seed, integrator="leapfrog", ensemble="nvt")]
    if k == "point":
        return [_nacl(case["natom"], seed, integrator="vv", ensemble="nve")]
    if k == "water":
        return [_water(case["nside"], seed)]
    if k == "pme":
        a = _nacl(case["natom"], seed, integrator="vv", ensemble="nve")
        a.update(lkspace=2, alfa=float(np.float32(3.09 / math.sqrt(a["rcutsq"]))), dt=1.0)
        return [a]
    if k == "npt":
        return [_nacl(case["natom"], seed, integrator="leapfrog", ensemble="npt")]
    if k == "fp64":
        return [_nacl(case["natom"], seed, integrator="vv", ensemble="nve")]
    rng = np.random.default_rng(seed + 1)
    sizes = _replica_sizes(case) if k == "replicas" else [case["natom"]] * case["nrep"]
    out = []
    for r, n in enumerate(sizes):
        out.append(synth.to_arrays(synth.nacl_replica(
            n, seed=seed * 1009 + r, eps_scale=tuple(rng.uniform(0.9, 1.1, 2)),
            sig_scale=tuple(rng.uniform(0.95, 1.05, 2)), charge_scale=float(rng.uniform(0.9, 1.1)),
            nmaxlist=416)))
    return out


NPT = dict(press_bar=1.0, tau_p_fs=1000.0)
ADJ = dict(w_pe=1.0, w_rdf=1.0, rdf_types=(0, 1), nbins=100, dr=0.05, sigma=0.05)


def _pinned(a):
    t = torch.empty(np.asarray(a).shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    t.numpy()[...] = a
    return t


class State:
    pass


def prepare(case, seed):
    st = State()
    st.case = case
    systems = _systems(case, seed)
    k = case["kind"]
    a = systems[0]
    if k in ("replicas", "adjoint"):
        st.sim = md.MDSystem.from_batch(systems)
        st.box = np.concatenate([np.broadcast_to(s["box"], (len(s["itype"]), 3)) for s in systems]).astype(np.float32)
    else:
        st.sim = md.MDSystem.from_arrays(**a)
        st.box = np.asarray(a["box"], np.float32)
    st.start = np.concatenate([s["pos"] for s in systems])
    if case.get("tuned"):   # tuned once on a copy of the run, the choice applied to the run
        with md.MDSystem.from_arrays(**a) as t:
            t.autotune()
            i = t.info()
        st.sim.set_tuning(i["pair_tpa"], i["list_tpa"], i["pair_depth"])
        st.sim.set_fused_step(i["fused_step"])
        st.sim.set_graph_rebuild(i["rebuild_inline"])
    if k == "pme":
        st.sim.set_pme(case["grid"])
    elif k == "npt":
        st.sim.set_barostat(**NPT)
    elif k == "fp64":
        st.sim.set_precision(64)
        st.start = st.start.astype(np.float64)
        st.box = st.box.astype(np.float64)
    elif k == "host":
        st.keep = [_pinned(a["pos"]), _pinned(a["vel"])]
        st.pos, st.vel = (t.numpy() for t in st.keep)
    elif k == "point":   # the next configurations to evaluate
        rng = np.random.default_rng(seed + 2)
        x = a["pos"].astype(np.float64)
        L = np.asarray(a["box"], np.float64)
        st.confs = []
        for _ in range(2):
            y = x + rng.uniform(-0.1, 0.1, x.shape)
            y -= L * np.floor(y / L + 0.5)
            st.confs.append(np.clip(y, -0.5 * L, 0.5 * L))
    return st


def _near_start(st, p):
    p -= st.box * np.rint((p - st.start) / st.box)
    return p


def run(st):
    c, sim = st.case, st.sim
    k = c["kind"]
    f32 = np.float32
    if k == "host":
        p, v, rec = sim.run_host(st.pos, st.vel, c["steps"], inplace=True, raw_records=True)
        return {"pos": _near_start(st, p.astype(f32)), "vel": v.astype(f32), "temper": rec["temper"].astype(f32)}
    if k == "point":
        out = []
        for x in st.confs:
            sim.set_positions(x)
            sim.compute_forces(md.TERM_ALL, energy=True)
            out.append({"force": sim.forces().astype(f32), "energy": sim.energies().astype(f32)})
        return out
    if k == "adjoint":
        o = sim.adjoint(c["steps"], checkpoint=c["checkpoint"], **ADJ)
        return {n: np.ascontiguousarray(o[n][:, :2, :2] if o[n].ndim == 3 else o[n]).astype(f32) for n in sorted(o)}
    sim.step(c["steps"], c.get("energy_every", 0))
    if k == "fp64":
        return {"pos": _near_start(st, sim.positions()), "vel": sim.velocities()}
    out = {"pos": sim.positions().astype(f32), "vel": sim.velocities().astype(f32)}
    if k == "npt":
        out["box"], out["pressure"] = (a.astype(f32) for a in sim.replica_boxes())
        out["pos"] -= out["box"] * np.rint(out["pos"] / out["box"] - st.start / st.box)
    else:
        _near_start(st, out["pos"])
    if k == "argon":   # energies of the run's last record (0 where it computed none)
        t = sim.thermo()
        out["temper"], out["pe"] = t["temper"], t["pe"]
    elif k == "replicas":
        out["ke"] = np.array([t["ke"] for t in sim.replica_thermo()], f32)
    return out


# ---- what a pass cannot do without ----

def _counts(case):
    """(atoms, unique pairs inside rc) of a case, from sizes and densities."""
    k = case["kind"]
    if k == "argon":
        n = 4 * case["ncell"] ** 3
        return n, n * 0.8442 * 4.0 / 3.0 * math.pi * 2.5 ** 3 / 2
    if k == "water":
        n = 3 * case["nside"] ** 3
        return n, n * 0.0999 * 4.0 / 3.0 * math.pi * 10.0 ** 3 / 2
    rho = 1.5 / ((22.98977 + 35.4527) / 2.0) * 0.602214076

    def pairs(n):
        rc = min(12.0, 0.4995 * (n / rho) ** (1.0 / 3.0) - 1.0)
        return n * rho * 4.0 / 3.0 * math.pi * rc ** 3 / 2

    if k == "replicas":
        sides = [m for m in range(8, 22, 2) if m ** 3 <= case["nmax"]]
        f = case["nrep"] / len(sides)
        return int(f * sum(m ** 3 for m in sides)), f * sum(pairs(m ** 3) for m in sides)
    n = case["natom"] * case.get("nrep", 1)
    return n, case.get("nrep", 1) * pairs(case["natom"])


def work(case):
    n, p = _counts(case)
    k = case["kind"]
    evals = {"point": 2, "adjoint": 3 * case.get("steps", 1)}.get(k, case.get("steps", 1))
    per_pair = 35.0 if k == "argon" else 60.0
    flops = evals * (p * per_pair + n * 30.0)
    if k == "water":
        flops += evals * n * 60.0
    if k == "pme":
        g = case["grid"] ** 3
        flops += evals * (n * 64 * 12.0 + 2 * 2.5 * g * math.log2(g))
    if k == "adjoint":
        return {"bytes": n * 48.0 + case["nrep"] * (100 + 13) * 4.0, "flops": flops}
    if k == "point":
        return {"bytes": 2 * n * (24.0 + 40.0), "flops": flops}
    return {"bytes": n * 96.0, "flops": flops}


# ---- the same results in 64 bits, with plain torch ----

DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a, dt=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), device=DEV).to(dt)


class Plain:
    """Systems (concatenated) in 64 bits: pair lists by brute force, LJ + Wolf /
    reaction field / Ewald real-space forces, harmonic bonds and angles."""

    def __init__(self, systems, pme_grid=0):
        cat = lambda f: np.concatenate([f(s) for s in systems])
        n = [len(s["itype"]) for s in systems]
        self.first = np.concatenate([[0], np.cumsum(n)])
        per = lambda v: _t(np.repeat(np.asarray(v, np.float64), n, axis=0))
        self.box = per([s["box"] for s in systems])
        self.rep = _t(np.repeat(np.arange(len(n)), n), torch.int64)
        self.ty = _t(cat(lambda s: s["itype"]), torch.int64)
        self.q = _t(cat(lambda s: s["charge"]))
        self.m = _t(cat(lambda s: np.asarray(s["type_mass"], np.float64)[s["itype"]]))
        self.nt = len(systems[0]["type_mass"])
        self.l1 = _t(np.stack([np.asarray(s["lj1"], np.float64) for s in systems]))
        self.l2 = _t(np.stack([np.asarray(s["lj2"], np.float64) for s in systems]))
        self.kind = systems[0]["lkspace"]
        rc2 = np.array([np.float64(np.float32(s["rcutsq"])) for s in systems])
        al = np.array([np.float64(np.float32(s["alfa"])) for s in systems])
        rc = np.sqrt(rc2)
        self.rc2, self.al, self.rc = _t(rc2), _t(al), _t(rc)
        self.krf = float(np.float32(systems[0]["reacf"]))
        ec = self._erfc(self.al * self.rc) * torch.exp(-(self.al * self.rc) ** 2)
        self.spi = 2.0 / math.sqrt(math.pi) * self.al
        on = 1.0 if self.kind == 1 else 0.0
        self.W = on * (ec / self.rc + self.spi * torch.exp(-(self.al * self.rc) ** 2))
        self.ucc = on * ec / self.rc if self.kind else 1.0 / self.rc + 0.5 * self.krf * self.rc2
        self.skin = float(systems[0]["skin"])
        self.bonds = self.angles = None
        if systems[0].get("bonds") is not None:
            s = systems[0]
            self.bonds, self.angles = _t(s["bonds"], torch.int64), _t(s["angles"], torch.int64)
            self.bp = [_t(np.float32(s[x])) for x in ("bnd1", "bnd2", "ang1", "ang2")]
        self.grid = pme_grid

    @staticmethod
    def _erfc(x):
        """A&S 7.1.26 without its exponential."""
        t = 1.0 / (1.0 + P_S * x)
        return ((((A_S[4] * t + A_S[3]) * t + A_S[2]) * t + A_S[1]) * t + A_S[0]) * t

    def pairs(self, x, margin, directed=False):
        """Atom pairs (i < j, or both ways) within rc + margin."""
        out = []
        for r, (a, b) in enumerate(zip(self.first[:-1], self.first[1:])):
            rmax = float(self.rc[r]) + margin
            rows = max(1, int(6e7) // int(b - a))
            L = self.box[int(a)]
            xa = x[int(a):int(b)]
            for i0 in range(0, int(b - a), rows):
                d2 = 0.0
                for k in range(3):
                    d = xa[i0:i0 + rows, None, k] - xa[None, :, k]
                    d -= L[k] * torch.round(d / L[k])
                    d2 = d2 + d * d
                i, j = torch.nonzero(d2 < rmax * rmax, as_tuple=True)
                i = i + i0
                keep = (i != j) if directed else (i < j)
                out.append(torch.stack([i[keep] + int(a), j[keep] + int(a)]))
        p = torch.cat(out, 1)
        if self.bonds is not None:   # bonded pairs are excluded
            n = len(self.q)
            b = self.bonds[:, 1:]
            ex = torch.cat([b[:, 0] * n + b[:, 1], b[:, 1] * n + b[:, 0]])
            p = p[:, ~torch.isin(p[0] * n + p[1], ex)]
        return p

    def diff(self, x, i, j):
        d = x[i] - x[j]
        L = self.box[i]
        return d - L * torch.round(d / L)

    def pair(self, x, ij, energy=False, l1=None, l2=None, s=None):
        """(i, j, d, r^2, F/r of the pair, its energy) of the pairs inside rc."""
        i, j = ij
        d = self.diff(x, i, j)
        r2 = (d * d).sum(1)
        keep = r2.detach() <= self.rc2[self.rep[i]]
        i, j, d, r2 = i[keep], j[keep], d[keep], r2[keep]
        R = self.rep[i]
        qq = QFAC * self.q[i] * self.q[j]
        if s is not None:
            qq = qq * s[R] ** 2
        r = torch.sqrt(r2)
        if self.kind == 0:
            ff = qq * (1.0 / r - self.krf * r2) / r2
            u = qq * (1.0 / r + 0.5 * self.krf * r2 - self.ucc[R]) if energy else None
        else:
            x_ = self.al[R] * r
            e = torch.exp(-x_ * x_)
            E = self._erfc(x_) * e
            ff = qq * (E / r + self.spi[R] * e - self.W[R]) / r2
            u = qq * (E / r - self.ucc[R] + self.W[R] * torch.log(r / self.rc[R])) if energy else None
        l1 = (self.l1 if l1 is None else l1)[R, self.ty[i], self.ty[j]]
        l2 = (self.l2 if l2 is None else l2)[R, self.ty[i], self.ty[j]]
        i6 = 1.0 / r2 ** 3
        ff = ff + (l1 * i6 - l2) * i6 / r2
        if energy:
            c6 = 1.0 / self.rc2[R] ** 3
            u = u + l1 / 12.0 * (i6 * i6 - c6 * c6) - l2 / 6.0 * (i6 - c6)
        return i, j, d, r2, ff, u

    def forces(self, x, ij):
        """Forces, and the sum of ff r^2 over unique pairs (and bonds)."""
        i, j, d, r2, ff, _ = self.pair(x, ij)
        F = torch.zeros_like(x)
        f = ff[:, None] * d
        F.index_add_(0, i, f)
        F.index_add_(0, j, -f)
        if self.bonds is not None:
            t, i, j = self.bonds.T
            d = self.diff(x, i, j)
            r = d.norm(dim=1)
            f = (self.bp[0][t] * (self.bp[1][t] / r - 1.0))[:, None] * d
            F.index_add_(0, i, f)
            F.index_add_(0, j, -f)
            t, i, c, j = self.angles.T
            a, b = self.diff(x, i, c), self.diff(x, j, c)
            na, nb = a.norm(dim=1, keepdim=True), b.norm(dim=1, keepdim=True)
            co = ((a * b).sum(1, keepdim=True) / (na * nb)).clamp(-0.9999999, 0.9999999)
            g = (self.bp[2][t][:, None] * (torch.acos(co) - self.bp[3][t][:, None])) / torch.sqrt(1.0 - co * co)
            fa = g * (b / nb - co * a / na) / na
            fb = g * (a / na - co * b / nb) / nb
            F.index_add_(0, i, fa)
            F.index_add_(0, j, fb)
            F.index_add_(0, c, -fa - fb)
        if self.grid:
            F = F + self.recip(x)
        return F, (ff * r2).sum()

    def recip(self, x):
        """Smooth particle-mesh Ewald forces, cubic B-splines."""
        K, L = self.grid, float(self.box[0, 0])
        al, V = float(self.al[0]), float(self.box[0].prod())
        u = K * torch.remainder((x + 0.5 * L) / L, 1.0)
        i0 = torch.floor(u)
        w = u - i0
        v = 1.0 - w
        th = torch.stack([v ** 3 / 6, (3 * w ** 3 - 6 * w ** 2 + 4) / 6, (-3 * w ** 3 + 3 * w ** 2 + 3 * w + 1) / 6,
                          w ** 3 / 6], -1)
        dt = torch.stack([-0.5 * v ** 2, 1.5 * w ** 2 - 2 * w, -1.5 * w ** 2 + w + 0.5, 0.5 * w ** 2], -1)
        ix = (i0.long()[..., None] - 3 + torch.arange(4, device=x.device)) % K
        at = ((ix[:, 0, :, None, None] * K + ix[:, 1, None, :, None]) * K + ix[:, 2, None, None, :]).reshape(len(x), 64)
        prod = lambda a, b, c: (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(len(x), 64)
        Q = torch.zeros(K ** 3, dtype=x.dtype, device=x.device)
        Q.index_add_(0, at.reshape(-1), (self.q[:, None] * prod(th[:, 0], th[:, 1], th[:, 2])).reshape(-1))
        mf = torch.fft.fftfreq(K, 1.0 / K, device=x.device, dtype=x.dtype)
        mh = torch.arange(K // 2 + 1, device=x.device, dtype=x.dtype)
        mod = lambda m: ((2.0 + torch.cos(2 * math.pi * m / K)) / 3.0) ** 2
        m2 = (mf[:, None, None] ** 2 + mf[None, :, None] ** 2 + mh[None, None, :] ** 2) / (L * L)
        m2[0, 0, 0] = 1.0
        infl = torch.exp(-math.pi ** 2 * m2 / (al * al)) / (
            math.pi * V * m2 * mod(mf)[:, None, None] * mod(mf)[None, :, None] * mod(mh)[None, None, :])
        infl[0, 0, 0] = 0.0
        conv = torch.fft.irfftn(torch.fft.rfftn(Q.view(K, K, K)) * infl, s=(K, K, K)) * float(K ** 3)
        c = conv.reshape(-1)[at]
        g = torch.stack([(c * prod(dt[:, 0], th[:, 1], th[:, 2])).sum(1), (c * prod(th[:, 0], dt[:, 1], th[:, 2])).sum(1),
                         (c * prod(th[:, 0], th[:, 1], dt[:, 2])).sum(1)], 1)
        return -QFAC * self.q[:, None] * (K / L) * g

    def energies(self, x, ij):
        i, j, _, _, _, u = self.pair(x, ij, energy=True)
        e = torch.zeros(len(x), dtype=x.dtype, device=x.device)
        e.index_add_(0, i, 0.5 * u)
        e.index_add_(0, j, 0.5 * u)
        return e


def _plain_steps(case, systems):
    """The case's steps in 64 bits: (x next to its start, v, per-step
    temperatures, box edge scale, pressure of the last step)."""
    s = systems[0]
    P = Plain(systems, case.get("grid", 0))
    x = _t(np.concatenate([a["pos"] for a in systems]))
    v = _t(np.concatenate([a["vel"] for a in systems]))
    m, dt, n = P.m[:, None], float(np.float32(s["dt"])), len(x)
    ndf = 3 * n - 3
    t0, tau = float(np.float32(s["temper_0"])), float(np.float32(s["tau_t"]))
    ke2 = lambda: (m * v * v).sum()
    kt = ndf * RGAS * t0
    Q = kt * tau * tau
    lam, xi, mu, scale, temps, press = 1.0, 0.0, 1.0, 1.0, [], 0.0
    ij = None
    leap = s["integrator"] == md.MD_LEAPFROG
    every, margin = (8, 1.5) if case["kind"] != "argon" else (16, 0.6)

    def F(x, step):
        nonlocal ij
        if ij is None or step % every == 0:
            ij = P.pairs(x, margin)
        return P.forces(x, ij)

    f, w = F(x, 0)
    for step in range(case["steps"]):
        if leap:
            if step:
                f, w = F(x, step)
            v = (v + f * dt / m) * lam
            x = x + v * dt
            T = float(ke2()) / (ndf * RGAS)
            temps.append(T)
            if s["enstype"] == 2:
                V = float(P.box[0].prod())
                press = (T * ndf * RGAS + float(w)) / (3.0 * V)
                x = x * mu
                P.box = P.box * mu
                scale *= mu
                k = 4.5e-5 * BAR * dt / (3.0 * NPT["tau_p_fs"])
                mu = min(max(1.0 - k * (NPT["press_bar"] / BAR - press), 1.0 - 1e-4), 1.0 + 1e-4)
            lam = math.sqrt(1.0 + dt / tau * (t0 / T - 1.0)) if s["enstype"] >= 1 else 1.0
            continue
        if s["integrator"] == md.MD_NH:
            k2 = float(ke2())
            xi += 0.25 * dt * (k2 - kt) / Q
            s1 = math.exp(-0.5 * dt * xi)
            xi += 0.25 * dt * (k2 * s1 * s1 - kt) / Q
            v = v * s1
        v = v + f * dt / (2.0 * m)
        x = x + v * dt
        f, w = F(x, step + 1)
        v = v + f * dt / (2.0 * m)
        if s["integrator"] == md.MD_NH:
            k2 = float(ke2())
            xi += 0.25 * dt * (k2 - kt) / Q
            s2 = math.exp(-0.5 * dt * xi)
            xi += 0.25 * dt * (k2 * s2 * s2 - kt) / Q
            v = v * s2
    return P, x, v, temps, scale, press


def _plain_adjoint(case, systems):
    P = Plain(systems)
    R, K = len(systems), case["steps"]
    x = _t(np.concatenate([a["pos"] for a in systems]))
    v = _t(np.concatenate([a["vel"] for a in systems]))
    m, dt = P.m[:, None], float(np.float32(systems[0]["dt"]))
    l1, l2 = P.l1.clone().requires_grad_(), P.l2.clone().requires_grad_()
    lns = torch.zeros(R, dtype=x.dtype, device=x.device, requires_grad=True)
    cnt = torch.bincount(P.rep, minlength=R).to(x.dtype)
    centre = (torch.arange(ADJ["nbins"], device=x.device, dtype=x.dtype) + 0.5) * ADJ["dr"]
    sg = ADJ["sigma"]
    rmax = ADJ["nbins"] * ADJ["dr"] + 5 * sg
    na = torch.zeros(R, dtype=x.dtype, device=x.device).index_add_(0, P.rep, (P.ty == 0).to(x.dtype))
    vol = P.box[_t(P.first[:-1], torch.int64)].prod(1)
    norm = vol[:, None] / (na * (cnt - na) * 4.0 * math.pi)[:, None] / centre ** 2

    def frame(x, ij):
        i, j, d, r2, ff, u = P.pair(x, ij, True, l1, l2, torch.exp(lns))
        F = torch.zeros_like(x).index_add(0, i, ff[:, None] * d)
        pe = torch.zeros(R, dtype=x.dtype, device=x.device).index_add(0, P.rep[i], 0.5 * u)
        sel = (P.ty[i] == 0) & (P.ty[j] == 1) & (r2.detach() < rmax * rmax)
        r, rep = torch.sqrt(r2[sel]), P.rep[i[sel]]
        b0 = torch.floor(r.detach() / ADJ["dr"]).long()
        h = torch.zeros(R * ADJ["nbins"], dtype=x.dtype, device=x.device)
        for o in range(-6, 7):
            b = b0 + o
            y = (b + 0.5) * ADJ["dr"] - r
            ok = (b >= 0) & (b < ADJ["nbins"]) & (y.detach().abs() <= 5 * sg)
            g = torch.exp(-0.5 * (y / sg) ** 2) / (math.sqrt(2 * math.pi) * sg)
            h = h.index_add(0, (rep * ADJ["nbins"] + b)[ok], g[ok])
        return F, pe, h.view(R, -1) * norm

    pe_sum, g_sum, ij = 0.0, 0.0, None
    for k in range(K + 1):
        if k % 8 == 0:
            ij = P.pairs(x.detach(), 1.5, directed=True)
        F, pe, g = frame(x, ij)
        pe_sum, g_sum = pe_sum + pe, g_sum + g
        if k:
            v = v + F * dt / (2.0 * m)
        if k < K:
            v = v + F * dt / (2.0 * m)
            x = x + v * dt
    gbar = g_sum / (K + 1)
    loss = ADJ["w_pe"] * pe_sum / (K + 1) / cnt + ADJ["w_rdf"] * (gbar ** 2).sum(1)
    d1, d2, ds = torch.autograd.grad(loss.sum(), [l1, l2, lns])
    return {n: t.detach().cpu().numpy() for n, t in
            (("loss", loss), ("gbar", gbar), ("dlj1", d1), ("dlj2", d2), ("dlns", ds))}


def exact(case, seed):
    k = case["kind"]
    systems = _systems(case, seed)
    n = sum(len(s["itype"]) for s in systems)
    if not torch.cuda.is_available() and n > 3000:
        return None
    if k == "point":
        st = None
        rng = np.random.default_rng(seed + 2)
        a = systems[0]
        x0, L = a["pos"].astype(np.float64), np.asarray(a["box"], np.float64)
        P, out = Plain(systems), []
        for _ in range(2):
            y = x0 + rng.uniform(-0.1, 0.1, x0.shape)
            y -= L * np.floor(y / L + 0.5)
            # the force kernels work on float32 positions
            y = _t(np.clip(y, -0.5 * L, 0.5 * L).astype(np.float32))
            ij = P.pairs(y, 0.1)
            i, j, d, r2, ff, _ = P.pair(y, ij)
            F = torch.zeros(len(y), 4, dtype=y.dtype, device=y.device)
            f = torch.cat([ff[:, None] * d, (ff * r2)[:, None]], 1)
            F.index_add_(0, i, f)
            f[:, :3] *= -1.0
            F.index_add_(0, j, f)
            out.append({"force": F.cpu().numpy(), "energy": P.energies(y, ij).cpu().numpy()})
        return out
    if k == "adjoint":
        return _plain_adjoint(case, systems)
    P, x, v, temps, scale, press = _plain_steps(case, systems)
    out = {"pos": x.cpu().numpy(), "vel": v.cpu().numpy()}
    if k == "host":
        out["temper"] = np.array(temps)
    elif k == "npt":
        out["box"] = np.asarray(systems[0]["box"], np.float64)[None, :] * scale
        out["pressure"] = np.array([press * BAR])
    elif k == "argon":
        out["temper"] = float((P.m[:, None] * v * v).sum()) / ((3 * len(v) - 3) * RGAS)
        out["pe"] = None
    elif k == "replicas":
        ke = torch.zeros(len(systems), dtype=x.dtype, device=x.device)
        out["ke"] = ke.index_add_(0, P.rep, 0.5 * (P.m[:, None] * v * v).sum(1)).cpu().numpy()
    return out
