"""Lanes split over clusters of 4, 8 and 16 CTAs (tis_params.launch_ctas),
through the C-ABI against the oracle: list sizes and lists bit-exact, forces
FP64 relative 1e-9 and mixed 1e-5 of max(|F_i|, median |F|), trajectories
with injected noise FP64 1e-8 A and mixed 1e-4 A, as for the other kernels.
Sizes at the edges of the division: CTAs without beads or items, bead counts
that are no multiple of 4, charged rows of 8, 16 and 32 threads, rows whose
partner lists do not fit shared memory, a periodic box, Ewald sums, Mg-P
tables and over-subscribed hydrogen-bond sites.  Every bead's sums run in
the same order whatever the number of CTAs, so these agree bit for bit."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

FORCE_TOL = {0: 1e-9, 1: 1e-5}
POS_TOL = {0: 1e-8, 1: 1e-4}


def chain(n):
    return synth.set_friction(synth.dt15_chain(n, 70 + n, hb_fraction=0.3), 0.5)


def system(kind):
    if kind.startswith("chain"):
        return chain(int(kind[5:])), synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0)
    if kind == "cadence":
        return chain(33), synth.dt15_params(ionic_strength=0.15, n_step_neighbor=10)
    if kind == "coulomb":
        return chain(33), synth.dt15_params(i_ele=3, cutoff_ele=60.0, n_step_neighbor=0)
    if kind == "none":
        return chain(33), synth.dt15_params(i_ele=0, n_step_neighbor=0)
    if kind == "pruned":
        base = synth.set_friction(synth.dt15_chain(22, 3, stem=6), 0.5)
        s = synth.duplicate_hbonds(synth.hairpin_coords(base, 6, seed=3), seed=4)
        return s, synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0)
    if kind == "tertiary":
        return synth.hairpin_tertiary(), synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0)
    if kind == "dt19":
        return synth.dt19_mg_system(), synth.dt19_params(i_periodic=1, psize=(80.0,) * 3, ionic_strength=0.05)
    if kind == "box":
        s = chain(22)
        s["xyz"] = s["xyz"] - s["xyz"].mean(axis=0) + np.array([35.0, -35.0, 0.0])   # across the box faces
        return s, synth.dt15_params(i_periodic=1, psize=(300.0, 260.0, 280.0), ionic_strength=0.15)
    assert kind == "ewald"
    s = chain(12)
    s["xyz"] = s["xyz"] - s["xyz"].mean(axis=0)
    s = synth.add_ions(s, 80.0, {"Mg": 4, "K": 20, "Cl": 28 - s["ncharge"]}, 5, clash=6.0)
    return s, synth.dt15_params(i_periodic=1, psize=(80.0,) * 3, i_ele=2, cutoff_ele=20.0, ewld_alpha=0.08, ewld_hmax=6.0)


def rel_force_err(f, ref):
    mag = np.linalg.norm(ref, axis=1)
    return np.max(np.linalg.norm(f - ref, axis=1) / np.maximum(mag, np.median(mag)))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["chain5", "chain22", "chain66", "chain162", "cadence", "coulomb", "none", "pruned",
                                  "tertiary", "dt19", "box", "ewald"])
def test_split_matches_oracle(tis_lib, kind, precision):
    s, par = system(kind)
    par = dict(par, precision=precision)
    temps, n, nsteps = [300.0, 320.0], s["nmp"], 12
    noise = np.random.default_rng(8).normal(size=(nsteps + 1, 2 * n, 3))
    u = np.random.default_rng(9).uniform(1e-6, 1.0, size=(2, 16384))
    orc = Oracle(s, dict(par, precision=0), temps)
    orc.set_state(np.tile(s["xyz"], (2, 1, 1)))
    orc.set_noise(noise.reshape(nsteps + 1, 2, n, 3), u)
    orc.time_integral_pre()
    fr = orc.force(2)[0] if kind != "pruned" else None   # (draws uniforms when it prunes)
    lists = orc.exv_list(2), orc.ele_list(2), orc.hb_list(2)
    orc.step(nsteps)
    xr = orc.get_state()[0].reshape(-1, 3)
    first = None
    for ctas in (4, 8, 16):
        eng = Engine([s], dict(par, launch_ctas=ctas), temps, nrep=[2])
        eng.set_state(np.tile(s["xyz"], (2, 1)))
        eng.set_noise(noise, u)
        eng.time_integral_pre()
        assert np.array_equal(eng.exv_list(2), lists[0])
        assert np.array_equal(eng.ele_list(2)[0], lists[1][0]) and np.array_equal(eng.ele_list(2)[1], lists[1][1])
        assert np.array_equal(eng.hb_list(2), lists[2])
        if fr is not None:
            assert rel_force_err(eng.force(2)[0], fr) < FORCE_TOL[precision]
        eng.step(5)
        eng.step(nsteps - 5)
        state = eng.get_state()
        assert np.abs(state[0] - xr).max() < POS_TOL[precision]
        if first is None:
            first = state
        for a, b in zip(first, state):
            assert np.array_equal(a, b), ctas
        eng.close()


@pytest.mark.parametrize("ctas", [8, 16])
def test_long_chain_with_and_without_partner_lists(tis_lib, ctas):
    """1,199 beads: the partner lists of a CTA's charged rows fit beside the
    rest on 16 CTAs, on 8 the rows' bits are read instead."""
    s = chain(400)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=1, launch_ctas=ctas)
    orc = Oracle(s, dict(par, precision=0, launch_ctas=0), [300.0])
    orc.set_state(s["xyz"][None])
    orc.neighbor()
    eng = Engine([s], par, [300.0])
    eng.set_state(s["xyz"])
    eng.neighbor()
    assert np.array_equal(eng.exv_list(), orc.exv_list()) and np.array_equal(eng.ele_list()[0], orc.ele_list()[0])
    assert rel_force_err(eng.force()[0], orc.force()[0]) < FORCE_TOL[1]
    eng.close()


def test_batch_with_some_lanes_split(tis_lib):
    """A batch whose long chains are split beside short ones on one CTA each:
    every chain's positions against the oracle's."""
    systems = [chain(k) for k in [300] * 12 + [20] * 150]
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=0)
    temps = [300.0] * len(systems)
    eng = Engine(systems, par, temps, nrep=[1] * len(systems))
    noise = np.random.default_rng(3).normal(size=(4, eng.nbead, 3))
    eng.set_state(np.vstack([s["xyz"] for s in systems]))
    eng.set_noise(noise)
    eng.time_integral_pre()
    eng.step(3)
    x = eng.get_state()[0]
    for k in (0, 11, 12, 161):
        s, lo = systems[k], eng.offsets[k]
        orc = Oracle(s, par, [300.0])
        orc.set_state(s["xyz"][None])
        orc.set_noise(noise[:, lo:lo + s["nmp"]].reshape(4, 1, s["nmp"], 3))
        orc.time_integral_pre()
        orc.step(3)
        assert np.abs(x[lo:lo + s["nmp"]] - orc.get_state()[0].reshape(-1, 3)).max() < POS_TOL[0]
        orc.close()
    eng.close()


@pytest.mark.parametrize("ctas,precision", [(2, 1), (4, 0), (8, 0), (16, 0), (8, 1)])
def test_near_lists_follow_beads_of_other_ctas(tis_lib, ctas, precision):
    """A dense chain over 300 steps, many near-list recordings: a contact with
    a bead that another CTA moves must not be missed.  Against one CTA per
    replica with the same noise (FP64: the same sums in another order; mixed:
    FP32 rounding, amplified over the run)."""
    s = synth.set_friction(synth.dt15_chain(40, 5, min_dist=2.8, confine=12.0), 0.5)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=precision)
    out = []
    for c in (1, ctas):
        eng = Engine([s], dict(par, launch_ctas=c), [400.0])
        eng.set_state(s["xyz"])
        eng.time_integral_pre()
        eng.step(300)
        out.append(eng.get_state()[0])
        eng.close()
    assert np.abs(out[0] - out[1]).max() < {0: 1e-6, 1: 1e-2}[precision]


@pytest.mark.parametrize("every,pair", [(0, False), (10, True), (43, True), (44, False)])
def test_short_rebuild_cadence_keeps_the_two_cta_kernel(tis_lib, every, pair):
    """64 replicas on two CTAs each: the split, or, with lists rebuilt often,
    the kernel whose rebuild is cheaper; both against one CTA per replica."""
    s = synth.set_friction(synth.dt15_chain(76, 5), 0.5)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=every, precision=1)
    out = []
    for extra in ({}, {"launch_ctas": 1}):
        eng = Engine([s], dict(par, **extra), list(np.geomspace(280.0, 400.0, 64)))
        if not extra:
            assert eng.status()["ctas_per_lane"] == (2 if pair else 1)
        eng.set_state(np.tile(s["xyz"], (64, 1)))
        eng.time_integral_pre()
        eng.step(12)
        out.append(eng.get_state()[0])
        eng.close()
    assert np.abs(out[0] - out[1]).max() < POS_TOL[1]
