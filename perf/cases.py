"""Workloads of the force-and-integrate engine, for timing and comparison.

Each case is one call sequence of a program that uses ``tis_b200.Engine``:

* ``point``    a single-point evaluation (lists, forces and energies of one
               structure), as an analysis or a force check does it;
* ``langevin`` a trajectory segment of one or several replicas of one chain
               (time_integral_pre, then steps, then the frame that is
               written), Debye-Hueckel electrostatics;
* ``hostloop`` the same driven by a host that calls one step at a time (the
               Fortran main loop);
* ``rex``      one period of temperature replica exchange;
* ``uneven``   a batch of independent chains of different length;
* ``ewald``    a chain with explicit ions in a periodic box, Ewald sums;
* ``bdhi``     Brownian dynamics with hydrodynamic interactions of bead
               chains (the diffusion tensor and its Cholesky factor
               refreshed every ``every`` steps).

The molecules are fixed by the case; the seed gives the thermal state (small
displacements, Maxwell velocities) and the noise key.  The FP64 option
returns the state as it is held; for the mixed option (FP32 forces) frames
are returned as the 32-bit numbers that trajectory files hold.

``exact`` evaluates the same model in 64 bits with plain torch: energies by
their formulas, forces by differentiation, the velocity-Verlet Langevin and
the Ermak-McCammon updates with the counter-based noise.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tis_b200 import synth
from tis_b200.engine import Engine

BOLTZ_J, N_AVO, KCAL = 1.38064852e-23, 6.022140857e23, 4184.0
KB = BOLTZ_J * (1.0 / KCAL * N_AVO)
ELE, EPS0 = 1.6021766208e-19, 8.854187817e-12


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a force check of one small hairpin: the smallest call, all latency
        dict(name="point_22nt_fp64", kind="point", nt=22, fp64=True),
        # the plain path: one small hairpin, FP64, a list every 10 steps
        dict(name="langevin_22nt_fp64", kind="langevin", nt=22, nrep=1, fp64=True, skin=False, ionic=0.150, steps=200),
        # one replica of a tRNA-sized chain, mixed precision, Verlet skin
        dict(name="langevin_76nt", kind="langevin", nt=76, nrep=1, fp64=False, skin=True, ionic=0.100, steps=100),
        # one medium chain in FP64
        dict(name="langevin_200nt_fp64", kind="langevin", nt=200, nrep=1, fp64=True, skin=True, ionic=0.150, steps=50),
        # one long chain, mixed precision
        dict(name="langevin_400nt", kind="langevin", nt=400, nrep=1, fp64=False, skin=True, ionic=0.150, steps=50),
        # a host that calls every step itself, a few replicas
        dict(name="hostloop_51nt_x8", kind="hostloop", nt=51, nrep=8, fp64=False, skin=True, ionic=0.150, steps=20),
        # temperature replica exchange, one period
        dict(name="rex_76nt_x64", kind="rex", nt=76, nrep=64, fp64=False, skin=True, ionic=0.100, steps=100),
        # independent chains of 20 to 400 nucleotides
        dict(name="uneven_x256", kind="uneven", nchain=256, lo=20, hi=400, fp64=False, skin=True, ionic=0.150, steps=30),
        # explicit Mg, K and Cl with Ewald sums, mixed precision
        dict(name="ewald_51nt_ions", kind="ewald", nt=51, box=150.0, fp64=False, skin=True, steps=20),
        # a smaller ion box in FP64
        dict(name="ewald_21nt_ions_fp64", kind="ewald", nt=21, box=95.0, fp64=True, skin=False, steps=20),
        # hydrodynamic interactions: a batch of bead chains, tensor-core factorisation, refresh every 10 steps
        dict(name="bdhi_x32", kind="bdhi", nchain=32, lo=100, hi=1000, fp64=False, every=10, steps=10),
        # hydrodynamic interactions in FP64, refreshed every step (the reference's rule)
        dict(name="bdhi_150_fp64", kind="bdhi", nchain=1, lo=150, hi=150, fp64=True, every=1, steps=4),
    ]


def _loguni(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["point", "langevin", "langevin", "langevin", "hostloop", "rex", "uneven", "ewald", "ewald",
                       "bdhi", "bdhi"])
    fp64 = rng.random() < 0.4
    skin = rng.random() < 0.7
    ionic = round(math.exp(rng.uniform(math.log(0.02), math.log(0.3))), 4)
    if kind == "point":
        return dict(kind=kind, nt=_loguni(rng, 8, 300), fp64=True)
    if kind in ("langevin", "hostloop", "rex"):
        nt = _loguni(rng, 8, 300 if fp64 else 400)
        nrep = _loguni(rng, 2 if kind == "rex" else 1, 64)
        steps = _loguni(rng, 20, 200) if kind != "hostloop" else rng.randint(3, 20)
        while nrep * (3 * nt) ** 2 * steps > 1.5e9:   # no more than the largest listed case
            if steps > 20:
                steps = max(20, steps // 2)
            else:
                nrep = max(2 if kind == "rex" else 1, nrep // 2)
                if nrep * (3 * nt) ** 2 * steps > 1.5e9 and nrep <= 2:
                    nt = max(8, nt // 2)
        return dict(kind=kind, nt=nt, nrep=nrep, fp64=fp64, skin=skin, ionic=ionic, steps=steps)
    if kind == "uneven":
        lo = _loguni(rng, 8, 60)
        return dict(kind=kind, nchain=_loguni(rng, 8, 200), lo=lo, hi=max(lo + 5, _loguni(rng, 60, 300)), fp64=fp64,
                    skin=skin, ionic=ionic, steps=rng.randint(10, 30))
    if kind == "ewald":
        nt = rng.randint(8, 51)
        return dict(kind=kind, nt=nt, box=round(rng.uniform(max(70.0, 40.0 + 1.5 * nt), 140.0), 1), fp64=fp64, skin=skin,
                    steps=rng.randint(5, 20))
    lo = _loguni(rng, 20, 300)
    hi = max(lo, _loguni(rng, 60, 500 if fp64 else 900))
    nchain = _loguni(rng, 1, 8 if fp64 else 28)
    return dict(kind="bdhi", nchain=nchain, lo=lo, hi=hi, fp64=fp64, every=rng.choice([1, 5, 10]) if hi < 300 else 10,
                steps=rng.choice([4, 10]))


# ----------------------------------------------------------------- inputs
# a regular duplex close to the model's natural bonds, angles, stacks and pairs: (radius, angle, height) of the
# phosphate, sugar and base of one strand (the other by the two-fold axis), twist and rise per pair
_HELIX = dict(P=(8.590, -4.2648, 5.352), S=(9.144, -3.7525, 4.517), B=(5.669, -3.4994, 2.114), twist=0.5630, rise=2.9135)


@functools.lru_cache(maxsize=None)
def _hairpin(nt, wseed):
    """A folded hairpin: a helical stem and a loop of 4 or 5 nucleotides on a half circle."""
    stem = max(1, (nt - 4) // 2)
    s = synth.set_friction(synth.dt15_chain(nt, wseed, stem=stem, min_dist=0.0), 0.5)
    x = {}
    for k in range(1, stem + 1):
        for kind in "PSB":
            r, ph, z = _HELIX[kind]
            for sign, n in ((1.0, k), (-1.0, nt + 1 - k)):
                a = sign * ph + _HELIX["twist"] * k
                x[kind, n] = np.array([r * math.cos(a), r * math.sin(a), sign * z + _HELIX["rise"] * k])
    a, b = x["S", stem], x["S", nt + 1 - stem]
    mid, u, up = 0.5 * (a + b), 0.5 * (a - b), np.array([0.0, 0.0, 1.0])
    up = up - u * (up @ u) / (u @ u)
    up *= np.linalg.norm(u) / np.linalg.norm(up)
    side = np.cross(u, up) / np.linalg.norm(np.cross(u, up))
    loop = nt - 2 * stem
    for q in range(1, loop + 2):
        th, tp = math.pi * q / (loop + 1), math.pi * (q - 0.5) / (loop + 1)
        out = math.cos(th) * u + math.sin(th) * up
        if q <= loop:
            x["S", stem + q] = mid + out
            x["B", stem + q] = mid + out * (1.0 + 4.7 / np.linalg.norm(out))
        x["P", stem + q] = mid + math.cos(tp) * u + math.sin(tp) * up + 3.2 * side
    order = [(kind, n) for n in range(1, nt + 1) for kind in ("SB" if n == 1 else "PSB")]
    return dict(s, xyz=np.array([x[key] for key in order]))


@functools.lru_cache(maxsize=None)
def _walk(nt, wseed):
    return synth.set_friction(synth.dt15_chain(nt, wseed, hb_fraction=0.3), 0.5)


@functools.lru_cache(maxsize=None)
def _ions(nt, box):
    s = _hairpin(nt, nt)
    s = dict(s, xyz=s["xyz"] - s["xyz"].mean(axis=0))
    litre = box ** 3 * 1e-27 * N_AVO
    n_mg, n_k = int(round(0.005 * litre)), int(round(0.150 * litre))
    n_k = max(n_k, s["ncharge"] - 2 * n_mg)
    return synth.add_ions(s, box, {"Mg": n_mg, "K": n_k, "Cl": 2 * n_mg + n_k - s["ncharge"]}, nt + 100, clash=6.0)


def _lengths(case):
    rng = np.random.default_rng(case["nchain"] * 1009 + case["lo"])
    if case["kind"] == "uneven":
        return np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), size=case["nchain"])).round().astype(int)
    return rng.integers(case["lo"], case["hi"] + 1, size=case["nchain"])


@functools.lru_cache(maxsize=None)
def _bead_chain(n, wseed):
    return synth.bead_chain(n, wseed)


def _inputs(case, seed):
    """(systems, parameters, temperatures, x, v) of a case: the molecules of
    the case in the thermal state of the seed."""
    kind, prec = case["kind"], 0 if case["fp64"] else 1
    cadence = 0 if case.get("skin") else 10
    if kind == "bdhi":
        systems = [_bead_chain(int(n), 11 + k) for k, n in enumerate(_lengths(case))]
        par = synth.bdhi_params(precision=prec, n_step_hydro=case["every"], seed=1000 + seed)
        temps, nrep = [300.0] * len(systems), [1] * len(systems)
    elif kind == "ewald":
        systems, temps, nrep = [_ions(case["nt"], case["box"])], [300.0], [1]
        par = synth.dt15_params(i_periodic=1, psize=(case["box"],) * 3, i_ele=2, cutoff_ele=20.0, ewld_alpha=0.05,
                                ewld_hmax=10.0, ionic_strength=0.165, precision=prec, n_step_neighbor=cadence,
                                seed=1000 + seed)
    else:
        if kind == "uneven":
            systems = [_walk(int(n), 40 + k) for k, n in enumerate(_lengths(case))]
            temps, nrep = [300.0] * len(systems), [1] * len(systems)
        else:
            nt = case["nt"]
            systems = [_hairpin(nt, nt) if nt <= 100 else _walk(nt, nt)]
            n = case.get("nrep", 1)
            temps = synth.temperature_ladder(n) if kind == "rex" else [300.0] * n
            nrep = [n]
        par = synth.dt15_params(ionic_strength=case.get("ionic", 0.150), precision=prec, n_step_neighbor=cadence,
                                seed=1000 + seed)
    rng = np.random.default_rng(seed)
    xs, vs, lane = [], [], 0
    for s, r in zip(systems, nrep):
        for _ in range(r):
            sd = 0.01 if kind == "bdhi" else 0.05
            xs.append(s["xyz"] + rng.normal(0.0, sd, size=s["xyz"].shape))
            vs.append(rng.normal(size=s["xyz"].shape) * np.sqrt(KB * temps[lane] / s["cmass"])[:, None])
            lane += 1
    return systems, par, temps, nrep, np.concatenate(xs), np.concatenate(vs)


# ------------------------------------------------------------------- calls
def prepare(case, seed):
    systems, par, temps, nrep, x, v = _inputs(case, seed)
    return dict(case=case, eng=Engine(systems, par, temps, nrep=nrep), x=x, v=v)


def run(state):
    case, eng = state["case"], state["eng"]
    kind = case["kind"]
    if kind == "point":
        eng.set_state(state["x"], state["v"])
        eng.neighbor()
        f, _ = eng.force(1)
        return dict(f=f, e=eng.energy(1))
    eng.set_step(0)
    eng.set_state(state["x"], state["v"])
    eng.time_integral_pre()
    if kind == "rex":
        eng.run(1, case["steps"], exchange=True)
    elif kind == "hostloop":
        for _ in range(case["steps"]):
            eng.step(1)
    else:
        eng.step(case["steps"])
    x, v, a = eng.get_state()
    if kind == "bdhi":   # no velocities on this path
        return dict(x=x if case["fp64"] else x.astype(np.float32))
    out = dict(x=x, v=v, a=a)
    return out if case["fp64"] else {k: q.astype(np.float32) for k, q in out.items()}


# -------------------------------------------------------------------- work
@functools.lru_cache(maxsize=None)
def _sizes(key):
    case = dict(key)
    systems, _, _, nrep, x, _ = _inputs(case, 0)
    return [(s["nmp"], s["ncharge"], s["nst"], s["nhb"], s["nba"], s["nbd"], r) for s, r in zip(systems, nrep)], len(x)


def work(case):
    sizes, nbead = _sizes(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    steps = case.get("steps", 1)
    table = sum(40 * n + 24 * bd + 28 * ba + 84 * st + 128 * hb for n, q, st, hb, ba, bd, r in sizes)
    if case["kind"] == "bdhi":
        refresh = -(-steps // case["every"])
        flops = sum(refresh * ((3 * n) ** 3 / 3 + 30 * n * n) + steps * (3 * (3 * n) ** 2 + 10 * n * n)
                    for n, *_ in sizes)
        return dict(bytes=48 * nbead + sum(16 * n for n, *_ in sizes), flops=flops)
    flops = 0.0
    for n, q, st, hb, ba, bd, r in sizes:
        # contact pairs of a bead are few; every charge pair within the cutoff, the bonded terms and the update
        per = 20 * q * (q - 1) / 2 + 200 * n + 300 * st + 500 * hb + 60 * ba + 20 * bd
        if case["kind"] == "ewald":
            per += 2 * 14 * q * 4168 + 12 * q * 33
        flops += r * steps * per
    return dict(bytes=(72 + 72) * nbead + table, flops=flops)


# ------------------------------------------------------------------- exact
def _philox(c, k0, k1):
    M = 0xFFFFFFFF
    c0, c1, c2, c3 = c
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57   # 64-bit products (wrap is the product modulo 2^64)
        h0, l0, h1, l1 = (p0 >> 32) & M, p0 & M, (p1 >> 32) & M, p1 & M
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c0, c1, c2, c3


def _noise(seed, lane, bead, istep):
    """Gaussian triple of every bead (counter-based Philox4x32-10, Box-Muller)."""
    M = 0xFFFFFFFF
    z = torch.zeros_like(bead)
    k0 = ((seed & M) ^ ((0x9E3779B9 * (lane + 1)) & M)) & M
    o = _philox((z + (istep & M), z + (istep >> 32), bead, z + 0x4E4F4953), k0, z + ((seed >> 32) & M))
    u = [((q >> 8) + 1).double() * 2.0 ** -24 for q in o]
    r1, r2 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    t1, t2 = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
    return torch.stack([r1 * torch.cos(t1), r1 * torch.sin(t1), r2 * torch.cos(t2)], dim=1)


def _dih(a, b, c):
    """atan2 dihedral of the vectors a, b, c as the stack and hbond terms take it."""
    m, n = torch.linalg.cross(a, b), torch.linalg.cross(b, c)
    return torch.atan2((a * n).sum(1) * b.norm(dim=1), (m * n).sum(1))


def _wrap(d):
    return d - 2.0 * math.pi * torch.round(d / (2.0 * math.pi))


def _angle(a, b):
    return torch.acos((a * b).sum(1) / (a.norm(dim=1) * b.norm(dim=1)))


class _Model:
    """Lanes of DT15 chains in 64 bits: bonded terms over all beads, pairs in
    padded groups of lanes of similar size."""

    def __init__(self, systems, par, temps, nrep):
        self.dev = dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        lanes = [s for s, r in zip(systems, nrep) for _ in range(r)]
        off = np.concatenate([[0], np.cumsum([s["nmp"] for s in lanes])])
        self.par, self.off, self.box = par, off, float(par["psize"][0]) if par["i_periodic"] else 0.0
        T = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=dt, device=dev)  # noqa: E731
        cat = lambda f: T(np.concatenate([np.asarray(f(s, k), dtype=np.float64) for k, s in enumerate(lanes)]))  # noqa: E731
        idx = lambda key, w: T(np.concatenate([np.asarray(s[key]).reshape(-1, w) - 1 + off[k] for k, s in enumerate(lanes)]),  # noqa: E731
                               torch.int64)
        self.temps = temps
        self.mass = cat(lambda s, k: s["cmass"])
        self.fric = cat(lambda s, k: s["fric"])
        self.temp = cat(lambda s, k: np.full(s["nmp"], temps[k]))
        self.lane = cat(lambda s, k: np.full(s["nmp"], k)).long()
        self.bead = torch.arange(int(off[-1]), device=dev)
        self.bd, self.ba = idx("ibd2mp", 2), idx("iba2mp", 3)
        self.st, self.hb = idx("idtrna_st2mp", 7), idx("idtrna_hb2mp", 6)
        self.bdn, self.bdk = cat(lambda s, k: s["bd_nat"]), cat(lambda s, k: s["coef_bd"])
        self.ban, self.bak = cat(lambda s, k: s["ba_nat"]), cat(lambda s, k: s["coef_ba"])
        self.stn, self.stk = cat(lambda s, k: s["dtrna_st_nat"].reshape(-1, 3)), cat(lambda s, k: s["coef_dtrna_st"].reshape(-1, 3))
        self.u0 = cat(lambda s, k: -s["dtrna_st_hsTm"].reshape(-1, 3)[:, 0] + KB * (temps[k] - s["dtrna_st_hsTm"].reshape(-1, 3)[:, 2])
                      * s["dtrna_st_hsTm"].reshape(-1, 3)[:, 1])
        self.hbn, self.hbk = cat(lambda s, k: s["dtrna_hb_nat"].reshape(-1, 6)), cat(lambda s, k: s["coef_dtrna_hb"].reshape(-1, 7))
        # groups of lanes for the pair terms
        self.groups = []
        order = sorted(range(len(lanes)), key=lambda k: -lanes[k]["nmp"])
        while order:
            n0 = lanes[order[0]]["nmp"]
            g = [order.pop(0)]
            while order and lanes[order[0]]["nmp"] >= 0.8 * n0 and len(g) < max(1, int(1.0e8 // n0 ** 2)):
                g.append(order.pop(0))
            self.groups.append(self._group([lanes[k] for k in g], [off[k] for k in g], [temps[k] for k in g], n0))

    def _group(self, lanes, offs, temps, n0):
        dev, par, B = self.dev, self.par, len(lanes)
        pad = lambda v: torch.as_tensor(v, device=dev)  # noqa: E731
        at = np.zeros((B, n0), dtype=np.int64)
        typ, cls = np.zeros((B, n0), dtype=np.int64), np.zeros((B, n0), dtype=np.int64)
        q, rad, eps = np.zeros((B, n0)), np.zeros((B, n0)), np.zeros((B, n0))
        for b, (s, o) in enumerate(zip(lanes, offs)):
            n = s["nmp"]
            at[b, :n] = o + np.arange(n)
            typ[b, :n] = s["imp2type"]
            for (lo, hi), c in zip(np.asarray(s["lunit2mp"]).reshape(-1, 2), s["iclass_unit"]):
                cls[b, lo - 1:hi] = c
            q[b, np.asarray(s["icharge2mp"]) - 1] = s["coef_charge"]
            rad[b, :n], eps[b, :n] = s["exv_radius"], s["exv_epsilon"]
        at, typ, cls, q, rad, eps = (pad(v) for v in (at, typ, cls, q, rad, eps))
        rna, live = cls == 2, cls > 0
        i, j = torch.arange(n0, device=dev)[:, None], torch.arange(n0, device=dev)[None, :]
        # local pairs of a chain: j < i + n_sep of the lower bead's type
        nsep = torch.where(typ == 2, par["n_sep_nlocal_P"], torch.where(typ == 4, par["n_sep_nlocal_S"], par["n_sep_nlocal_B"]))
        low = torch.where((i < j)[None], nsep[:, :, None], nsep[:, None, :])
        ok = live[:, :, None] & live[:, None, :] & (i != j)[None]
        ok &= ~(rna[:, :, None] & rna[:, None, :] & ((i - j).abs()[None] < low))
        dij = rad[:, :, None] + rad[:, None, :]
        dij = torch.where(rna[:, :, None] & rna[:, None, :], torch.full_like(dij, par["exv_dist"]), dij)
        dij = torch.where(ok, dij, torch.full_like(dij, -1.0))
        ek, coef, lam = zip(*(self._ele(t) for t in temps))
        return dict(at=at, live=live, dij=dij, eps=eps, q=q, coef=pad(np.array(coef)), lam=pad(np.array(lam)))

    def _ele(self, t):
        par = self.par
        tc = t - 273.15
        ek = 87.740 - 0.4008 * tc + 9.398e-4 * tc * tc - 1.410e-6 * tc ** 3 if par["i_diele"] else par["diele_water"]
        coef = (N_AVO / KCAL) * 1.0e10 * ELE * ELE / (4.0 * math.pi * EPS0 * ek)
        lam = 1.0e10 * math.sqrt(1.0e-3 * EPS0 * ek * BOLTZ_J / (2.0 * N_AVO * ELE * ELE)) * math.sqrt(t / par["ionic_strength"])
        return ek, coef, lam

    def _img(self, d):
        return d - self.box * torch.round(d / self.box) if self.box else d

    def smooth(self, X):
        """Energies of the bonds, stacks and hydrogen bonds (angles apart)."""
        d = lambda a, b: X[b] - X[a]  # noqa: E731
        bd, st, hb = self.bd, self.st, self.hb
        e_bd = (self.bdk * (d(bd[:, 0], bd[:, 1]).norm(dim=1) - self.bdn) ** 2).sum()
        v21, v34, v54 = d(st[:, 0], st[:, 1]), d(st[:, 3], st[:, 2]), d(st[:, 3], st[:, 4])
        v56, v76 = d(st[:, 5], st[:, 4]), d(st[:, 5], st[:, 6])
        ediv = 1.0 + self.stk[:, 0] * (v21.norm(dim=1) - self.stn[:, 0]) ** 2
        ediv = ediv + self.stk[:, 1] * _wrap(_dih(v34, v54, v56) - self.stn[:, 1]) ** 2
        n1 = -torch.linalg.cross(v54, v56)
        m1 = torch.linalg.cross(v76, v56)
        p2 = torch.atan2((v76 * n1).sum(1) * v56.norm(dim=1), (m1 * n1).sum(1))
        ediv = ediv + self.stk[:, 2] * _wrap(p2 - self.stn[:, 2]) ** 2
        e_st = (self.u0 / ediv).sum()
        g = lambda p, r: self._img(X[hb[:, p]] - X[hb[:, r]])  # noqa: E731
        v12, v13, v53, v42, v46 = g(0, 1), g(0, 2), g(4, 2), g(3, 1), g(3, 5)
        nat, cf = self.hbn, self.hbk
        dd = v12.norm(dim=1) - nat[:, 0]
        on = dd.abs() <= self.par["hb_cutoff_dist"]
        a1, a2 = _angle(v13, v12), _angle(v12, v42)
        c4212, c1213 = torch.linalg.cross(v42, v12), torch.linalg.cross(v12, v13)
        p0 = torch.atan2((v42 * c1213).sum(1) * v12.norm(dim=1), (c4212 * c1213).sum(1))
        n = -c1213
        pa = torch.atan2((v53 * n).sum(1) * v13.norm(dim=1), (torch.linalg.cross(v53, v13) * n).sum(1))
        m, c4246 = -c4212, torch.linalg.cross(v42, v46)
        pb = torch.atan2((v12 * c4246).sum(1) * v42.norm(dim=1), (m * c4246).sum(1))
        ex = cf[:, 1] * dd ** 2 + cf[:, 2] * (a1 - nat[:, 1]) ** 2 + cf[:, 3] * (a2 - nat[:, 2]) ** 2
        ex = ex + cf[:, 4] * _wrap(p0 - nat[:, 3]) ** 2 + cf[:, 5] * _wrap(pa - nat[:, 4]) ** 2 + cf[:, 6] * _wrap(pb - nat[:, 5]) ** 2
        e_hb = torch.where(on, cf[:, 0] * torch.exp(-ex), torch.zeros_like(ex)).sum()
        return e_bd, e_st, e_hb

    def force(self, x):
        X = x.detach().requires_grad_(True)
        E = sum(self.smooth(X))
        F = -torch.autograd.grad(E, X)[0]
        # angles: 2 k (theta - theta0) / sqrt(max(|u x v|^2, 1)) times the gradient of the dot product's ratio
        ba = self.ba
        u, v = x[ba[:, 1]] - x[ba[:, 0]], x[ba[:, 2]] - x[ba[:, 1]]
        c11, c22, c21 = (u * u).sum(1), (v * v).sum(1), (u * v).sum(1)
        th = torch.acos(torch.clamp(-c21 / torch.sqrt(c11 * c22), -1.0, 1.0))
        f = 2.0 * self.bak * (th - self.ban) / torch.sqrt(torch.clamp(c11 * c22 - c21 ** 2, min=1.0))
        fa, fb = f[:, None] * (u * (c21 / c11)[:, None] - v), f[:, None] * (v * (c21 / c22)[:, None] - u)
        F = F.index_add(0, ba[:, 0], -fa).index_add(0, ba[:, 1], fa - fb).index_add(0, ba[:, 2], fb)
        for g in self.groups:
            F = F.index_add(0, g["at"].reshape(-1), self._pairs(g, x).reshape(-1, 3))
        return F + self._recip(x) if self.par["i_ele"] == 2 else F

    def _geom(self, g, x):
        P = torch.where(g["live"][:, :, None], x[g["at"]], torch.full((), 1.0e6, dtype=x.dtype, device=x.device))
        d = [self._img(P[:, None, :, k] - P[:, :, None, k]) for k in range(3)]
        r2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        return d, torch.where(r2 == 0.0, torch.full_like(r2, 1.0e12), r2)

    def _pairs(self, g, x):
        par = self.par
        d, r2 = self._geom(g, x)
        r = torch.sqrt(r2)
        a = par["exv_adjust"]
        dr = r + a - g["dij"]
        ro2 = (a / dr) ** 2
        f = (12.0 * g["eps"][:, :, None] * g["eps"][:, None, :] * (ro2 ** 7 - ro2 ** 4) * dr / a ** 2 / r).abs()
        f = torch.where(r <= g["dij"], torch.clamp(f, max=50.0), torch.zeros_like(f))
        qq = g["q"][:, :, None] * g["q"][:, None, :] * g["coef"][:, None, None]
        if par["i_ele"] == 1:
            lam = g["lam"][:, None, None]
            e = torch.clamp(qq / r2 * (1.0 / r + 1.0 / lam) * torch.exp(-r / lam), max=50.0)
            f = f + torch.where(r <= par["cutoff_ele"] * lam, e, torch.zeros_like(e))
        elif par["i_ele"] == 2:
            al = par["ewld_alpha"]
            e = qq / r2 * (torch.erfc(al * r) / r + 2.0 * al / math.sqrt(math.pi) * torch.exp(-(al * r) ** 2))
            f = f + torch.where(r <= par["cutoff_ele"], e, torch.zeros_like(e))
        out = torch.stack([-(f * c).sum(2) for c in d], dim=2)
        return torch.where(g["live"][:, :, None], out, torch.zeros_like(out))

    def _kvec(self):
        h = int(math.ceil(self.par["ewld_hmax"]))
        k = torch.cartesian_prod(*[torch.arange(-h, h + 1, device=self.dev, dtype=torch.float64)] * 3)
        h2 = (k * k).sum(1)
        k = k[(h2 > 0) & (h2 <= self.par["ewld_hmax"] ** 2)] * (2.0 * math.pi / self.box)
        k2 = (k * k).sum(1)
        return k, 2.0 * math.pi / self.box ** 3 * torch.exp(-k2 / (4.0 * self.par["ewld_alpha"] ** 2)) / k2

    def _recip(self, x):
        F = torch.zeros_like(x)
        k, C = self._kvec()
        for g in self.groups:
            for b in range(g["at"].shape[0]):
                q = g["q"][b]
                at = g["at"][b][q != 0.0]
                q = q[q != 0.0]
                ph = x[at] @ k.T
                s, c = torch.sin(ph) * q[:, None], torch.cos(ph) * q[:, None]
                w = g["coef"][b] * 2.0 * C * (s * c.sum(0) - c * s.sum(0))
                F = F.index_add(0, at, w @ k)
        return F

    def energies(self, x, v):
        """The 25 energy components (E_TYPE) of lane 1."""
        par, e = self.par, torch.zeros(25, dtype=torch.float64, device=self.dev)
        e[1] = 0.5 * (self.mass * (v * v).sum(1)).sum()
        e[2], e[15], e[16] = self.smooth(x)
        u, w = x[self.ba[:, 0]] - x[self.ba[:, 1]], x[self.ba[:, 2]] - x[self.ba[:, 1]]
        e[3] = (self.bak * (_angle(u, w) - self.ban) ** 2).sum()
        g = self.groups[0]
        _, r2 = self._geom(g, x)
        r = torch.sqrt(r2)
        ro6 = (par["exv_adjust"] / (r + par["exv_adjust"] - g["dij"])) ** 6
        ex = g["eps"][:, :, None] * g["eps"][:, None, :] * (ro6 * ro6 - 2.0 * ro6 + 1.0)
        ex = torch.where(r + par["exv_adjust"] - g["dij"] > par["exv_inf"], ex, torch.full_like(ex, 1.0e10))
        e[17] = 0.5 * torch.where(r <= g["dij"], ex, torch.zeros_like(ex)).sum()
        lam = g["lam"][:, None, None]
        el = g["q"][:, :, None] * g["q"][:, None, :] * g["coef"][:, None, None] / r * torch.exp(-r / lam)
        e[7] = 0.5 * torch.where(r <= par["cutoff_ele"] * lam, el, torch.zeros_like(el)).sum()
        e[0] = e[2:].sum()
        return e

    def langevin(self, x, v, steps):
        dt, seed = self.par["tstep"], self.par["seed"]
        c1 = torch.sqrt(2.0 * self.fric * KB * self.temp / (dt * self.mass))[:, None]
        h = 0.5 * dt * self.fric
        u1, u2 = 1.0 - h, 1.0 - h + h * h
        c2, c3, c4 = (u1 * u2)[:, None], (0.5 * dt * u1)[:, None], (dt * u1)[:, None]
        acc = lambda x, k: self.force(x) / self.mass[:, None] + c1 * _noise(seed, self.lane, self.bead, k)  # noqa: E731
        a = acc(x, 0)
        for k in range(1, steps + 1):
            x = x + (c4 * v + 0.5 * dt * dt * a)
            b = acc(x, k)
            v, a = c2 * v + c3 * (a + b), b
        return x, v, a


def _bd_force(s, x):
    d = x[1:] - x[:-1]
    r = d.norm(dim=1)
    dd = r - s["fene_nat"][0]
    f = (s["coef_fene"][0] * dd / (1.0 - dd * dd / s["dist2_fene"][0]) / r)[:, None] * d
    F = torch.zeros_like(x)
    F[:-1] += f
    F[1:] -= f
    w = x[None, :, :] - x[:, None, :]
    i = torch.arange(len(x), device=x.device)
    ro2 = s["wca_nat"][0] ** 2 / (w * w).sum(2).clamp(min=1.0e-12)
    on = ((i[:, None] - i[None, :]).abs() >= 2) & (ro2 >= 1.0)
    g = torch.clamp(12.0 * s["coef_wca"][0, 0] / s["wca_nat"][0] ** 2 * (ro2 ** 7 - ro2 ** 4), max=50.0)
    return F - (torch.where(on, g, torch.zeros_like(g))[:, :, None] * w).sum(1)


def _rpy(x, a, c6, c8):
    n = len(x)
    w = x[None, :, :] - x[:, None, :]
    r2 = (w * w).sum(2)
    eye = torch.eye(n, dtype=torch.bool, device=x.device)
    r2 = torch.where(eye, torch.ones_like(r2), r2)
    r = torch.sqrt(r2)
    p1 = torch.where(eye, torch.full_like(r, c6 / a), c8 / r * (1.0 + 2.0 * a * a / (3.0 * r2)))
    p2 = torch.where(eye, torch.zeros_like(r), c8 / r * (1.0 - 2.0 * a * a / r2) / r2)
    D = p2[:, :, None, None] * w[:, :, :, None] * w[:, :, None, :]
    D += p1[:, :, None, None] * torch.eye(3, dtype=x.dtype, device=x.device)
    return D.permute(0, 2, 1, 3).reshape(3 * n, 3 * n)


def _bd(systems, par, x, every, steps):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    kt, dt = KB * 300.0, par["tstep"]
    c6, c8 = kt / (6.0 * math.pi * par["viscosity"]), kt / (8.0 * math.pi * par["viscosity"])
    out, o = [], 0
    for lane, s in enumerate(systems):
        n = s["nmp"]
        X = torch.as_tensor(x[o:o + n], dtype=torch.float64, device=dev)
        bead = torch.arange(o, o + n, device=dev)
        lid = torch.full_like(bead, lane)
        F = _bd_force(s, X)
        for k in range(1, steps + 1):
            if (k - 1) % every == 0:
                D = _rpy(X, par["hi_radius"], c6, c8)
                L = torch.linalg.cholesky(D)
            xi = _noise(par["seed"], lid, bead, k).reshape(-1)
            X = X + (dt / kt * (D @ F.reshape(-1)) + math.sqrt(2.0 * dt) * (L @ xi)).reshape(-1, 3)
            F = _bd_force(s, X)
        out.append(X.cpu().numpy())
        o += n
    return np.concatenate(out)


def exact(case, seed):
    systems, par, temps, nrep, x, v = _inputs(case, seed)
    if case["kind"] == "bdhi":
        return dict(x=_bd(systems, par, x, case["every"], case["steps"]))
    m = _Model(systems, par, temps, nrep)
    X, V = (torch.as_tensor(q, dtype=torch.float64, device=m.dev) for q in (x, v))
    if case["kind"] == "point":
        return dict(f=m.force(X).cpu().numpy(), e=m.energies(X, V).cpu().numpy())
    X, V, A = m.langevin(X, V, case["steps"])
    # the velocities of a replica exchange are rescaled by decisions that have no value of their own
    return dict(x=X.cpu().numpy(), v=None if case["kind"] == "rex" else V.cpu().numpy(), a=A.cpu().numpy())
