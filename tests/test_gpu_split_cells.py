"""Bonds, angles and stacks of lanes split over clusters in a periodic box:
they belong to the unwrapped positions (force_bond.F90:41-47,
force_bangle.F90:103-115, force_dtrna_stack.F90:60-90), hydrogen bonds and
tertiary stacks to the nearest image (force_dtrna_hbond15.F90:91-110).  The
kernel holds wrapped positions and each bead's cell, against the oracle:
chains given broken across the box faces and several boxes away, and beads
that cross faces between rebuilds of one call.  Forces FP64 relative 1e-9 and
mixed 1e-5 of max(|F_i|, median |F|), positions 1e-8 and 1e-4 A, as for every
kernel."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

BOX = np.array([260.0, 220.0, 240.0])
FORCE_TOL = {0: 1e-9, 1: 1e-5}
POS_TOL = {0: 1e-8, 1: 1e-4}


def chain(shift):
    s = synth.set_friction(synth.dt15_chain(22, 5, hb_fraction=0.3), 0.5)
    s["xyz"] = s["xyz"] - s["xyz"].mean(axis=0) + np.array(shift) * BOX
    return s


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ctas", [4, 8])
@pytest.mark.parametrize("start", ["whole", "wrapped", "far", "apart"])
def test_forces_of_unwrapped_bonds(tis_lib, start, ctas, precision):
    s = chain((0.5, -0.5, 0.5))
    x = s["xyz"].copy()
    if start == "wrapped":
        x -= BOX * np.round(x / BOX)
    elif start == "far":
        x += BOX * np.array([3.0, -2.0, 600.0])
    elif start == "apart":
        x[len(x) // 2:] += BOX * np.array([1.0, 0.0, -1.0])
    par = synth.dt15_params(i_periodic=1, psize=tuple(BOX), ionic_strength=0.15, precision=precision)
    orc = Oracle(s, dict(par, precision=0), [300.0])
    eng = Engine([s], dict(par, launch_ctas=ctas), [300.0])
    orc.set_state(x[None])
    eng.set_state(x)
    for _ in range(2):   # lists from unwrapped positions, then from the wrapped ones
        orc.neighbor()
        eng.neighbor()
        ref, f = orc.force()[0], eng.force()[0]
        mag = np.linalg.norm(ref, axis=1)
        assert np.max(np.linalg.norm(f - ref, axis=1) / np.maximum(mag, np.median(mag))) < FORCE_TOL[precision]
    eng.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("every", [0, 5])
def test_beads_that_cross_faces(tis_lib, every, precision):
    """A chain that flies through three faces, lists rebuilt meanwhile."""
    s = chain((0.45, -0.45, 0.45))
    par = synth.dt15_params(i_periodic=1, psize=tuple(BOX), ionic_strength=0.15, precision=precision,
                            n_step_neighbor=every)
    steps, n = 40, s["nmp"]
    v = np.tile(np.array([20.0, -20.0, 20.0]), (n, 1))
    noise = np.random.default_rng(2).normal(size=(steps + 1, n, 3))
    orc = Oracle(s, dict(par, precision=0), [300.0])
    orc.set_state(s["xyz"][None], v[None])
    orc.set_noise(noise[:, None])
    orc.time_integral_pre()
    orc.step(steps)
    ref = orc.get_state()[0].reshape(-1, 3)
    cells = np.round((ref - orc.get_pxyz().reshape(-1, 3)) / BOX)
    assert len({tuple(c) for c in cells}) > 1
    for ctas in (4, 8):
        eng = Engine([s], dict(par, launch_ctas=ctas), [300.0])
        eng.set_state(s["xyz"], v)
        eng.set_noise(noise)
        eng.time_integral_pre()
        eng.step(steps // 2)
        eng.step(steps // 2)
        assert np.abs(eng.get_state()[0] - ref).max() < POS_TOL[precision]
        eng.close()
