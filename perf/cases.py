"""Performance cases of the DPD engine: runs as a user's program makes them, through the
public entry points (Engine, Batch, the C ABI's state and AoS calls).

A case names a system of `gpumdpd_b200.inputs` with its sizes and options:

  plain     single-species fluid, fix nve                       (Engine)
  melt      A5B5 diblock chains, harmonic bonds                 (Engine, fp32 or fp64)
  slab      many-body DPD liquid slab with its vapour           (Engine)
  angles    chains with harmonic bonds and angles               (Engine)
  channel   liquid between a frozen and a moving particle wall  (Engine; move, two_wall)
  sweep     uneven A/B replicas with an A-B RDF compute         (Batch)
  plugin    one timestep of a host MD loop on its own AoS device buffers
            (fix nve, pair and bond forces)                     (Engine.*_aos)

A pass advances the system by `steps` timesteps and hands back the state and the thermo
rows of those steps, as a program does that samples a trajectory.  The single-precision
engine's results are handed on as float32, the FP64 engine's as float64.
"""
import ctypes
import math

import numpy as np
import torch

from gpumdpd_b200 import Batch, Engine, capi, inputs



def listed():
    return [
        # the smallest system a box of 3 cells of the reference's default cutoff holds,
        # advanced one step at a time by a program that looks at every step
        {"name": "plain_192_single_step", "kind": "plain", "L": 4.0, "skin": 0.3, "dt": 0.04, "steps": 1},
        # the textbook Groot-Warren fluid (3000 particles): small systems, many steps
        {"name": "plain_3k", "kind": "plain", "L": 10.0, "skin": 0.3, "dt": 0.02, "steps": 20},
        # a copolymer melt of workstation size, and one where the list lives several steps
        {"name": "melt_24k", "kind": "melt", "L": 20.0, "skin": 0.3, "dt": 0.02, "steps": 20},
        {"name": "melt_192k", "kind": "melt", "L": 40.0, "skin": 0.3, "dt": 0.01, "steps": 40},
        # the production melt (3 million beads) at the skin the tuner picks for it, sampled
        # for transport coefficients: velocities and forces
        {"name": "melt_3M", "kind": "melt", "L": 100.0, "skin": 0.0, "dt": 0.01, "steps": 30, "positions": False},
        # many-body DPD: liquid slab, density pass and force pass
        {"name": "slab_384k", "kind": "slab", "Lx": 40.0, "Lz": 120.0, "skin": 0.3, "dt": 0.01, "steps": 14},
        # semiflexible chains: angles beside pairs and bonds
        {"name": "angles_24k", "kind": "angles", "L": 20.0, "skin": 0.3, "dt": 0.02, "steps": 20},
        # Couette flow between particle walls: group fixes in the step
        {"name": "channel_21k", "kind": "channel", "L": 16.0, "Lz": 28.0, "skin": 0.3, "dt": 0.02, "steps": 20},
        # a parameter sweep: uneven replicas packed into one engine, RDF sampled
        {"name": "sweep_48", "kind": "sweep", "replicas": 48, "Lmin": 8.0, "Lmax": 24.0, "skin": 0.3, "dt": 0.01,
         "steps": 20},
        # the double-precision engine on a small and on a large system
        {"name": "fp64_3k", "kind": "melt", "fp64": True, "L": 10.0, "skin": 0.3, "dt": 0.02, "steps": 20},
        {"name": "fp64_192k", "kind": "melt", "fp64": True, "L": 40.0, "skin": 0.3, "dt": 0.02, "steps": 20},
        # the plugins inside another program's loop: one timestep on that program's buffers
        {"name": "plugin_81k", "kind": "plugin", "L": 30.0, "skin": 0.3, "dt": 0.02, "steps": 1},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["plain", "plain", "melt", "melt", "melt", "slab", "angles", "channel", "sweep", "fp64", "plugin"])
    # trajectories of the same inputs part with time: a pass stays where they can be compared
    span = 0.14 if kind == "slab" else 0.3
    c = {"kind": kind, "skin": rng.choice([0.0, 0.3, 0.3]), "dt": 0.01 if kind == "slab" else rng.choice([0.01, 0.02, 0.04])}
    c["steps"] = min(rng.choice([1, 10, 20, 40]), int(span / c["dt"] + 1e-9))
    if kind == "plain":
        c["L"] = round(_log(rng, 4.0, 45.0), 3)
    elif kind == "melt":
        c["L"] = round(_log(rng, 8.0, 75.0), 3)
    elif kind == "slab":
        c.update(Lx=round(_log(rng, 8.0, 40.0), 3), Lz=round(_log(rng, 24.0, 120.0), 3))
    elif kind == "angles":
        c["L"] = round(_log(rng, 6.0, 40.0), 3)
    elif kind == "channel":
        c.update(L=round(_log(rng, 6.0, 30.0), 3), Lz=round(_log(rng, 12.0, 40.0), 3))
    elif kind == "sweep":
        c.update(replicas=rng.randint(2, 64), Lmin=round(rng.uniform(5.0, 8.0), 3), Lmax=round(rng.uniform(9.0, 24.0), 3))
    elif kind == "fp64":
        c.update(kind="melt", fp64=True, L=round(_log(rng, 5.0, 42.0), 3))
    else:
        c.update(L=round(_log(rng, 6.0, 60.0), 3), steps=1)
    return c


def _systems(case, seed):
    """The case's systems (one, or a sweep's replicas)."""
    kind, dt, skin = case["kind"], case["dt"], case["skin"]
    every = max(1, case["steps"] // 2)  # two thermo rows a pass
    kw = dict(dt=dt, skin=skin, thermo=every)
    if kind in ("melt", "angles", "plugin") and skin == 0.0:
        kw["max_rho"] = 15.0  # random-walk chains start with a few dense spots: room for 64 neighbours
    if kind == "plain":
        return [inputs.plain_dpd(L=case["L"], seed=seed, **kw)]
    if kind in ("melt", "plugin"):
        return [inputs.diblock_melt(L=case["L"], seed=seed, **kw)]
    if kind == "slab":
        Lz = case["Lz"]
        return [inputs.mdpd_slab(Lx=case["Lx"], Ly=case["Lx"], Lz=Lz, z0=Lz / 3.0, z1=2.0 * Lz / 3.0, seed=seed, **kw)]
    if kind == "angles":
        return [inputs.angle_chains(L=case["L"], seed=seed, **kw)]
    if kind == "channel":
        return [inputs.wall_channel(L=case["L"], Lz=case["Lz"], seed=seed, **kw)]
    n = case["replicas"]
    out = []
    for r in range(n):  # sizes spread over the range, out of order
        u = (r * 0.6180339887498949) % 1.0
        L = case["Lmin"] * (case["Lmax"] / case["Lmin"]) ** u
        out.append(inputs.binary_mixture(L, 25.0 + 20.0 * r / max(n - 1, 1), seed=(seed * 64 + r) % (1 << 40),
                                         rdf=(min(3.0, 0.5 * L), 150, 100), **kw))
    return out


def _rows(case):
    return 2 if case["steps"] > 1 else 1


class _Frame:
    """Host buffers a sampling program keeps: positions, velocities, images, forces by tag."""

    def __init__(self, n):
        self.x, self.v, self.f = (np.empty((n, 3)) for _ in range(3))
        self.image = np.empty((n, 3), dtype=np.int32)


def prepare(case, seed):
    systems = _systems(case, seed)
    s = systems[0]
    if case["kind"] == "sweep":
        batch = Batch([q.run_in for q in systems], [q.c_system() for q in systems])
        off = np.concatenate([[0], np.cumsum([q.n for q in systems])])
        box = np.concatenate([np.broadcast_to(q.box, (q.n, 3)) for q in systems])
        return {"case": case, "batch": batch, "frame": _Frame(int(off[-1])), "off": off,
                "box": torch.from_numpy(np.ascontiguousarray(box))}
    eng = Engine(s.run_in, system=s.c_system(), precision="fp64" if case.get("fp64") else "fp32")
    if case["kind"] != "plugin":
        return {"case": case, "engine": eng, "frame": _Frame(s.n), "box": torch.tensor(np.ascontiguousarray(s.box))}
    # the host program's device buffers, with the forces of step 0 in them
    dev = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", t)  # noqa: E731
    st = {"case": case, "engine": eng, "n": s.n, "nb": len(s.bonds), "step": 0, "pos": dev(s.x, torch.float32),
          "uw": dev(s.x, torch.float32), "vel": dev(s.v, torch.float32), "force": torch.zeros(s.n, 3, device="cuda"),
          "id": torch.arange(1, s.n + 1, dtype=torch.int32, device="cuda"), "type": dev(s.types, torch.int32),
          "bonds": dev(s.bonds, torch.int32), "group": torch.arange(s.n, dtype=torch.int32, device="cuda")}
    _plugin_forces(st)
    return st


def _plugin_forces(st):
    p = lambda k: st[k].data_ptr()  # noqa: E731
    st["engine"].pair_compute_aos(p("pos"), p("vel"), p("id"), p("type"), st["n"], st["step"], p("force"))
    st["engine"].bond_compute_aos(p("pos"), p("bonds"), st["nb"], p("force"))


def _thermo(t):
    energy = np.column_stack([t["pair_pe"], t["bond_pe"], t["angle_pe"], t["ke"]])
    return energy, np.column_stack([t["temp"], t["p"]])


def run(state):
    case = state["case"]
    if case["kind"] == "plugin":
        p = lambda k: state[k].data_ptr()  # noqa: E731
        e, n = state["engine"], state["n"]
        state["step"] += 1
        e.nve_aos(0, p("group"), n, p("type"), p("pos"), p("uw"), p("vel"), p("force"))
        _plugin_forces(state)
        e.nve_aos(1, p("group"), n, p("type"), p("pos"), p("uw"), p("vel"), p("force"))
        return {"x": state["uw"], "v": state["vel"], "f": state["force"]}
    fr, lib = state["frame"], capi.load()
    if case["kind"] == "sweep":
        b, off = state["batch"], state["off"]
        b.run(case["steps"])
        thermo = []
        for r in range(b.n):
            i, j = off[r], off[r + 1]
            if lib.dpd_batch_get_state(b.h, r, *(capi.ptr(q[i:j]) for q in (fr.x, fr.v, fr.image, fr.f))):
                raise RuntimeError("state of replica %d" % r)
            thermo.append(_thermo(b.thermo(r, _rows(case))))
        energy, press = (np.concatenate([t[k] for t in thermo]) for k in (0, 1))
    else:
        e = state["engine"]
        e.run(case["steps"])
        where = capi.ptr(fr.x), capi.ptr(fr.image)
        if not case.get("positions", True):
            where = None, None
        if lib.dpd_get_state(e.h, where[0], capi.ptr(fr.v), where[1], capi.ptr(fr.f)):
            raise RuntimeError("state")
        energy, press = _thermo(e.thermo(_rows(case)))
    out = {"v": torch.from_numpy(fr.v), "f": torch.from_numpy(fr.f), "energy": torch.from_numpy(energy),
           "pressure": torch.from_numpy(press)}
    if case.get("positions", True):
        # unwrapped: what displacements, chain vectors and spectra are taken from
        out["x"] = torch.from_numpy(fr.x) + torch.from_numpy(fr.image) * state["box"]
    return out if case.get("fp64") else {k: q.float() for k, q in out.items()}


def _count(case):
    """(particles, bonds, angles) of a case, a sweep's in the mean."""
    kind = case["kind"]
    if kind == "slab":
        return 2.0 * case["Lx"] ** 2 * case["Lz"], 0, 0
    if kind == "channel":
        return 3.0 * case["L"] ** 2 * case["Lz"], 0, 0
    if kind == "sweep":
        a, b = case["Lmin"] ** 3, case["Lmax"] ** 3
        return case["replicas"] * 3.0 * (b - a) / math.log(b / a), 0, 0
    n = 3.0 * case["L"] ** 3
    if kind == "plain":
        return n, 0, 0
    return n, 0.9 * n, 0.8 * n if kind == "angles" else 0


def work(case):
    """Per timestep: position, velocity and force of every particle in and out once (the
    bond and angle tables in); the force of every pair inside the cutoff, with the integer
    operations of its random number counted as operations."""
    n, bonds, angles = _count(case)
    rho = 6.0 if case["kind"] == "slab" else 3.0
    word = 8 if case.get("fp64") else 4
    pairs = n * rho * 2.0 * math.pi / 3.0
    return {"bytes": case["steps"] * (2 * 9 * word * n + 12 * bonds + 16 * angles),
            "flops": case["steps"] * (pairs * (190.0 if case["kind"] != "slab" else 215.0) + 40.0 * bonds + 120.0 * angles + 20.0 * n)}


# --- the same in plain torch, 64 bits -------------------------------------------------
_M = 0xFFFFFFFF


def _asr(v, k):
    return (((v ^ 0x80000000) - 0x80000000) >> k) & _M


def _saru(s1, s2, seed, step):
    """The 32 random bits of a pair (int64 tensors holding uint32 values).  Both precisions of
    the engine take the stream through a float, so theta is made from float(bits)."""
    s3 = (seed + step) & _M
    s3 = s3 ^ (((s1 << 7) & _M) ^ (s2 >> 6))
    s2 = (s2 + ((s1 >> 4) ^ (s3 >> 15))) & _M
    s1 = s1 ^ ((((s2 << 9) & _M) + ((s3 << 8) & _M)) & _M)
    s3 = s3 ^ ((0xA5366B4D * ((s2 >> 11) ^ ((s1 << 1) & _M))) & _M)
    s2 = (s2 + 0x72BE1579 * (((s1 << 4) & _M) ^ (s3 >> 16))) & _M
    s1 = s1 ^ ((0x3F38A6ED * ((s3 >> 5) ^ _asr(s2, 22))) & _M)
    s2 = (s2 + s1 * s3) & _M
    s1 = (s1 + (s3 ^ (s2 >> 2))) & _M
    s2 = s2 ^ _asr(s2, 17)
    st = (0x79DEDEA3 * (s1 ^ _asr(s1, 14))) & _M
    w = ((st + s2) & _M) ^ _asr(st, 8)
    st = (st + w * (w ^ 0xDDDF97F5)) & _M
    w = (0xABCB96F7 + (w >> 1)) & _M
    total = 0
    for _ in range(8):
        total = (total + 0x9E3779B9) & _M
        st = (st + ((((w << 4) + 0xA341316C) & _M) ^ ((w + total) & _M) ^ (((w >> 5) + 0xC8013EA4) & _M))) & _M
        w = (w + ((((st << 4) + 0xAD90777D) & _M) ^ ((st + total) & _M) ^ (((st >> 5) + 0x7E95761E) & _M))) & _M
    v = ((st ^ (st >> 26)) + w) & _M
    return ((v ^ (v >> 20)) * 0x6957F5A7) & _M


class _Exact:
    """Packed systems advanced in FP64: cell search, pair, bond and angle forces,
    velocity Verlet, fix move and two_wall (the channel's)."""

    def __init__(self, case, systems):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, k=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=k, device=dev)  # noqa: E731
        self.case, self.dev, self.nrep = case, dev, len(systems)
        ns = [s.n for s in systems]
        self.rep = t(np.repeat(np.arange(len(ns)), ns), torch.int64)
        self.ns = t(ns)
        self.box = t([s.box for s in systems])
        single = case["kind"] == "plugin"  # the plugin's inputs are single precision
        cast = (lambda a: a.astype(np.float32).astype(np.float64)) if single else (lambda a: a)
        self.x = t(cast(np.concatenate([s.x for s in systems])))  # unwrapped
        self.v = t(cast(np.concatenate([s.v for s in systems])))
        self.type = t(np.concatenate([s.types for s in systems]), torch.int64) - 1
        self.tag = t(np.concatenate([np.arange(1, n + 1) for n in ns]), torch.int64)
        self.bonds = None if systems[0].bonds is None else t(systems[0].bonds, torch.int64) - 1
        self.angles = None if systems[0].angles is None else t(systems[0].angles, torch.int64) - 1
        # coefficients from the command text: pair_coeff i j A gamma, or i j A B gamma (mdpd)
        A, B, g, seed = [], [], [], []
        for s in systems:
            nt = len(s.masses)
            a3 = np.zeros((3, nt, nt))
            for line in s.run_in.splitlines():
                w = line.split()
                if w[0] == "pair_style":
                    self.mdpd, self.kT, self.rd = w[1] == "mdpd", float(w[2]), float(w[4]) if w[1] == "mdpd" else 1.0
                    seed.append(int(w[-1]))
                elif w[0] == "pair_coeff":
                    i, j, c = int(w[1]) - 1, int(w[2]) - 1, [float(q) for q in w[3:]]
                    val = (c[0], c[1], c[2]) if self.mdpd else (c[0], 0.0, c[1])
                    a3[:, i, j] = a3[:, j, i] = val
                elif w[0] == "bond_coeff":
                    self.bk, self.br0 = float(w[2]), float(w[3])
                elif w[0] == "angle_coeff":
                    self.ak, self.at0 = float(w[2]), math.radians(float(w[3]))
            A.append(a3[0]), B.append(a3[1]), g.append(a3[2])
        self.A, self.B, self.g, self.seed = t(A), t(B), t(g), t(seed, torch.int64)
        self.nc = torch.clamp((self.box).floor(), min=3).to(torch.int64)  # cells of the cutoff, 1
        cells = self.nc.prod(1)
        self.coff = torch.cumsum(cells, 0) - cells
        self.ncell = int(cells.sum())
        self.half = [(0, 0, 0)] + [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)
                                   if k > 0 or (k == 0 and (j > 0 or (j == 0 and i > 0)))]

    def pairs(self):
        """Index pairs within the cutoff and their displacements x_i - x_j."""
        b, nc = self.box[self.rep], self.nc[self.rep]
        xw = self.x - torch.floor(self.x / b) * b
        c = torch.minimum((xw / b * nc).to(torch.int64), nc - 1)
        lin = lambda q: self.coff[self.rep] + (q[:, 0] * nc[:, 1] + q[:, 1]) * nc[:, 2] + q[:, 2]  # noqa: E731
        key = lin(c)
        order = torch.argsort(key)
        cnt = torch.bincount(key, minlength=self.ncell)
        start = torch.cumsum(cnt, 0) - cnt
        rank = torch.empty_like(order)
        rank[order] = torch.arange(len(order), device=self.dev)
        m, n = int(cnt.max()), len(order)
        step = max(1, (24 << 20) // n)
        I, J, D = [], [], []
        for o in self.half:
            q = (c + torch.tensor(o, device=self.dev)) % nc
            nb = key if o == (0, 0, 0) else lin(q)
            first, num = start[nb], cnt[nb]
            for k0 in range(0, m, step):
                k = torch.arange(k0, min(m, k0 + step), device=self.dev)
                ok = k[None, :] < num[:, None]
                if o == (0, 0, 0):
                    ok &= first[:, None] + k[None, :] > rank[:, None]
                i, kk = torch.nonzero(ok, as_tuple=True)
                j = order[first[i] + k[kk]]
                d = xw[i] - xw[j]
                bi = b[i]
                d = d - torch.round(d / bi) * bi
                near = (d * d).sum(1) <= 1.0
                I.append(i[near]), J.append(j[near]), D.append(d[near])
        return torch.cat(I), torch.cat(J), torch.cat(D)

    def forces(self, step):
        f = torch.zeros_like(self.x)
        e = torch.zeros(self.nrep, 3, dtype=torch.float64, device=self.dev)
        vir = torch.zeros(self.nrep, 6, dtype=torch.float64, device=self.dev)

        def virial(rep, d, g):
            w = torch.stack([d[:, a] * g[:, b] for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], 1)
            vir.index_add_(0, rep, w)

        i, j, d = self.pairs()
        r = d.square().sum(1).sqrt()
        rep, ti, tj = self.rep[i], self.type[i], self.type[j]
        A, g = self.A[rep, ti, tj], self.g[rep, ti, tj]
        w = 1.0 - r
        bits = _saru(torch.minimum(self.tag[i], self.tag[j]), torch.maximum(self.tag[i], self.tag[j]), self.seed[rep], step)
        theta = math.sqrt(3.0) * (bits.float().double() * 2.0 ** -31 - 1.0)
        fp = A * w - g * w * w * (d * (self.v[i] - self.v[j])).sum(1) / r
        fp += torch.sqrt(g * (2.0 * self.kT / self.case["dt"])) * w * theta
        pe = 0.5 * A * w * w
        if self.mdpd:
            wd = torch.clamp(1.0 - r / self.rd, min=0.0)
            rho = torch.zeros(len(self.x), dtype=torch.float64, device=self.dev)
            add = 15.0 / (2.0 * math.pi * self.rd ** 3) * wd * wd
            rho.index_add_(0, i, add).index_add_(0, j, add)
            both = self.B[rep, ti, tj] * (rho[i] + rho[j])
            fp += both * wd
            pe = pe + 0.25 * self.rd * both * wd * wd
        gvec = d * (fp / r)[:, None]
        f.index_add_(0, i, gvec).index_add_(0, j, -gvec)
        e[:, 0].index_add_(0, rep, pe)
        virial(rep, d, gvec)
        near = lambda q: q - torch.round(q / self.box[0]) * self.box[0]  # noqa: E731
        if self.bonds is not None:
            i, j = self.bonds[:, 1], self.bonds[:, 2]
            d = near(self.x[i] - self.x[j])
            r = d.square().sum(1).sqrt()
            gvec = d * (-2.0 * self.bk * (r - self.br0) / r)[:, None]
            f.index_add_(0, i, gvec).index_add_(0, j, -gvec)
            e[0, 1] += (self.bk * (r - self.br0) ** 2).sum()
            virial(self.rep[i], d, gvec)
        if self.angles is not None:
            i, j, k = self.angles[:, 1], self.angles[:, 2], self.angles[:, 3]
            d1, d2 = near(self.x[i] - self.x[j]), near(self.x[k] - self.x[j])
            r1, r2 = d1.square().sum(1).sqrt(), d2.square().sum(1).sqrt()
            c = ((d1 * d2).sum(1) / (r1 * r2)).clamp(-1.0, 1.0)
            s = (torch.linalg.cross(d1, d2).square().sum(1).sqrt() / (r1 * r2))
            dth = torch.atan2(s, c) - self.at0
            a = -2.0 * self.ak * dth / s.clamp(min=0.001)
            a11, a12, a22 = a * c / r1 ** 2, -a / (r1 * r2), a * c / r2 ** 2
            fi, fk = a11[:, None] * d1 + a12[:, None] * d2, a22[:, None] * d2 + a12[:, None] * d1
            f.index_add_(0, i, fi).index_add_(0, k, fk).index_add_(0, j, -fi - fk)
            e[0, 2] += (self.ak * dth * dth).sum()
            virial(self.rep[i], d1, fi), virial(self.rep[i], d2, fk)
        return f, e, vir

    def thermo(self, e, vir):
        v = self.v
        kin = torch.zeros_like(vir)
        kin.index_add_(0, self.rep, torch.stack([v[:, a] * v[:, b] for a, b in
                                                 ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], 1))
        ke = 0.5 * (kin[:, 0] + kin[:, 3] + kin[:, 5])
        temp = 2.0 * ke / (3.0 * self.ns - 3.0)
        return torch.cat([e, ke[:, None]], 1), torch.cat([temp[:, None], (kin + vir) / self.box.prod(1)[:, None]], 1)

    def advance(self, steps, every):
        dt, rows = self.case["dt"], []
        moving = self.type == 2 if self.case["kind"] == "channel" else None
        nve = (self.type == 0)[:, None].double() if moving is not None else 1.0
        if moving is not None:
            lo, hi = self.x[self.type == 1, 2].max(), self.x[moving, 2].min()
        f, e, vir = self.forces(0)
        for n in range(1, steps + 1):
            self.v += nve * (0.5 * dt) * f
            self.x += nve * dt * self.v
            if moving is not None:
                V = torch.tensor([0.5, 0.0, 0.0], dtype=torch.float64, device=self.dev)
                self.v[moving] = V
                self.x[moving] += V * dt
                z, liquid = self.x[:, 2], self.type == 0
                for wall, out in ((lo, liquid & (z < lo)), (hi, liquid & (z > hi))):
                    self.x[out, 2] = 2.0 * wall - z[out]
                    self.v[out, 2] = -self.v[out, 2]
            f, e, vir = self.forces(n)
            self.v += nve * (0.5 * dt) * f
            if n % every == 0:
                rows.append(self.thermo(e, vir))
        return f, rows


def exact(case, seed):
    n = _count(case)[0]
    if n * case["steps"] > 4e7:
        return None
    systems = _systems(case, seed)
    ex = _Exact(case, systems)
    f, rows = ex.advance(case["steps"], max(1, case["steps"] // 2))
    host = lambda q: q.cpu()  # noqa: E731
    out = {"x": host(ex.x), "v": host(ex.v), "f": host(f)}
    if case["kind"] == "plugin":
        return out
    if not case.get("positions", True):
        del out["x"]
    rows = rows[-_rows(case):]
    # replica by replica, its rows in order of time
    out["energy"] = host(torch.stack([r[0] for r in rows], 1).reshape(-1, 4))
    out["pressure"] = host(torch.stack([r[1] for r in rows], 1).reshape(-1, 7))
    return out
