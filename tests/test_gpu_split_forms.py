"""Replicas split over 4, 8 and 16 CTAs against one CTA per replica on seeded
random systems of every form the kernels take: one to three chains (several
units), dense ones, hairpins, tertiary stacks, over-subscribed sites and ions;
open and periodic boxes, started anywhere; Debye-Hueckel, Coulomb, Ewald sums
or none; every rebuild rule and margin.  Lists, rebuild and clamp counts equal;
forces in FP64 relative 1e-9 of max(|F_i|, median |F|) and positions after 20
steps 1e-8 A, as for every kernel (other orders of the same sums); mixed
forces against one CTA's mixed ones within 1e-5 (both are within 1e-5 of FP64
where no bond is straight; here the two roundings are compared), or half of
what one CTA's differ from FP64 by, where that is more."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu

INDEX = ("icharge2mp", "ibd2mp", "iba2mp", "idtrna_st2mp", "idtrna_hb2mp", "lunit2mp")
COUNTS = ("nmp", "nunit", "ncharge", "nbd", "nba", "nst", "nhb", "nhbsite", "nfene", "nwca", "ntst")


def merge(a, b, shift):
    out = {}
    for k in set(a) | set(b):
        if k in COUNTS:
            out[k] = int(a.get(k, 0)) + int(b.get(k, 0))
            continue
        if k not in a or k not in b or np.ndim(a[k]) == 0:
            out[k] = a.get(k, b.get(k))
            continue
        x, y = np.asarray(a[k]), np.asarray(b[k])
        if k == "xyz":
            y = y + shift
        elif k in INDEX:
            y = y + a["nmp"]
        elif k == "idtrna_hb2hbsite":
            y = np.where(y > 0, y + a.get("nhbsite", 0), y)
        out[k] = np.concatenate([x, y]) if x.shape[1:] == y.shape[1:] else x
    return out


def draw(rng):
    def chain(n, **k):
        return synth.set_friction(synth.dt15_chain(n, int(rng.integers(1, 999)), hb_fraction=0.4, **k), 0.5)

    kind = rng.choice(["one", "two", "three", "dense", "hairpin", "tertiary", "ions", "sites"])
    nt = int(rng.integers(4, 45))
    if kind == "one":
        s = chain(nt)
    elif kind == "two":
        s = merge(chain(nt), chain(int(rng.integers(4, 30))), np.array([12.0, 5.0, 3.0]))
    elif kind == "three":
        s = merge(merge(chain(nt), chain(7), np.array([9.0, 4.0, 3.0])), chain(5), np.array([-7.0, 6.0, 9.0]))
    elif kind == "dense":
        s = chain(min(nt, 40), min_dist=2.8, confine=12.0)
    elif kind == "hairpin":
        s = synth.hairpin_coords(chain(22, stem=6), 6, seed=int(rng.integers(1, 99)))
    elif kind == "tertiary":
        s = synth.hairpin_tertiary(int(rng.integers(1, 60)))
    elif kind == "ions":
        s = synth.add_ions(chain(min(nt, 16)), 70.0, {"Mg": 3, "K": 12, "Cl": 6}, int(rng.integers(1, 99)), clash=5.0)
    else:
        s = synth.duplicate_hbonds(synth.hairpin_coords(chain(22, stem=6), 6, seed=3), seed=4)
    par = dict(ionic_strength=float(rng.uniform(0.02, 0.3)), n_step_neighbor=int(rng.choice([0, 1, 3, 7, 10])))
    ele = rng.choice(["dh", "none", "coulomb"] + (["ewald"] * 2 if kind == "ions" else []))
    periodic = kind == "ions" or bool(rng.integers(0, 2))
    if ele == "none":
        par["i_ele"] = 0
    elif ele == "coulomb":
        par.update(i_ele=3, cutoff_ele=float(rng.uniform(20.0, 60.0)))
    elif ele == "ewald":
        par.update(i_ele=2, ewld_alpha=0.15, ewld_hmax=float(rng.choice([4.0, 6.5, 9.0])), cutoff_ele=20.0)
    x = s["xyz"] + rng.normal(0.0, 0.05, size=s["xyz"].shape)
    if periodic:
        ext = float(np.ptp(x, axis=0).max())
        side = 70.0 if kind == "ions" else float(rng.uniform(max(60.0, 0.7 * ext), max(90.0, 2.0 * ext)))
        par.update(i_periodic=1, psize=(side,) * 3 if ele == "ewald" else (side, 1.1 * side, 0.95 * side))
        x = x + rng.uniform(-200.0, 200.0, size=3)
    if rng.integers(0, 3) == 0:
        par["neigh_margin"] = float(rng.uniform(2.0, 10.0))
    return s, synth.dt15_params(**par), x


def evaluate(s, par, x, v, noise, uniforms):
    eng = Engine([s], par, [300.0])
    eng.set_state(x, v)
    eng.set_noise(noise, uniforms)
    eng.neighbor()
    pairs, coef = eng.ele_list()
    lists = (eng.exv_list(), pairs, coef, eng.hb_list())
    f = eng.force()[0]
    eng.set_state(x, v)
    eng.time_integral_pre()
    eng.step(7)
    eng.step(13)
    st = eng.status()
    out = lists, f, eng.get_state()[0], (st["n_rebuild"], st["n_clamp"])
    eng.close()
    return out


@pytest.mark.parametrize("seed", range(24))
def test_split_is_the_one_cta_kernel(tis_lib, seed):
    rng = np.random.default_rng(100 + seed)
    s, par, x = draw(rng)
    v = rng.normal(0.0, 0.5, size=x.shape)
    noise, uniforms = rng.normal(size=(22, s["nmp"], 3)), rng.uniform(1e-6, 1.0, size=(1, 20000))
    lists, f, pos, counts = evaluate(s, dict(par, precision=0, launch_ctas=1), x, v, noise, uniforms)
    mag = np.linalg.norm(f, axis=1)
    scale = np.maximum(np.maximum(mag, np.median(mag)), 1.0e-12)
    mixed = evaluate(s, dict(par, precision=1, launch_ctas=1), x, v, noise, uniforms)[1]
    off = np.max(np.linalg.norm(mixed - f, axis=1) / scale)
    for ctas in (4, 8, 16):
        got = evaluate(s, dict(par, precision=0, launch_ctas=ctas), x, v, noise, uniforms)
        assert all(np.array_equal(p, q) for p, q in zip(got[0], lists))
        assert np.max(np.linalg.norm(got[1] - f, axis=1) / scale) < 1e-9
        assert np.abs(got[2] - pos).max() < 1e-8 and got[3] == counts
        got = evaluate(s, dict(par, precision=1, launch_ctas=ctas), x, v, noise, uniforms)
        assert all(np.array_equal(p, q) for p, q in zip(got[0], lists))
        assert np.max(np.linalg.norm(got[1] - mixed, axis=1) / scale) < max(1e-5, 0.5 * off)
