"""One CTA per replica (launch_ctas 1), asked for: the kernel that batches
filling the chip and every context with a launch field run, on the systems
where the library by itself now splits the replica.  Lists bit-exact, forces
FP64 relative 1e-9 and mixed 1e-5 of max(|F_i|, median |F|), trajectories
FP64 1e-8 A and mixed 1e-4 A against the oracle, as for every kernel; the
binned list build across a periodic box, also after skin rebuilds."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine
from oracle.oracle import Oracle
from test_gpu_cells import binned, compare_lists
from test_gpu_parity import SYSTEMS, rel_force_err

pytestmark = pytest.mark.gpu

FORCE_TOL = {0: 1e-9, 1: 1e-5}
POS_TOL = {0: 1e-8, 1: 1e-4}


def ewald_box():
    s = synth.set_friction(synth.dt15_chain(12, 3, stem=3), 0.5)
    return synth.add_ions(s, 40.0, {"Mg": 2, "K": 10, "Cl": 3}, 9, clash=5.0)


KINDS = dict(SYSTEMS, ewald=(ewald_box, dict(i_periodic=1, psize=(40.0,) * 3, i_ele=2, ewld_alpha=0.2, ewld_hmax=8.0,
                                             cutoff_ele=19.9)))


def case(name, precision):
    make, extra = KINDS[name]
    extra = dict(extra)
    base = extra.pop("_base", synth.dt15_params)
    s = make()
    par = base(**dict(dict(ionic_strength=0.15, n_step_neighbor=0, precision=precision), **extra))
    return s, par


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("name", list(KINDS))
def test_lists_forces_and_steps(tis_lib, name, precision):
    s, par = case(name, precision)
    n, steps = s["nmp"], 10
    noise = np.random.default_rng(6).normal(size=(steps + 1, n, 3))
    eng = Engine([s], dict(par, launch_ctas=1), [300.0])
    assert eng.launch()["layout"] == 1
    orc = Oracle(s, dict(par, precision=0), [300.0])
    eng.set_state(s["xyz"])
    orc.set_state(s["xyz"][None])
    eng.neighbor()
    orc.neighbor()
    compare_lists(eng, orc)
    assert np.array_equal(eng.hb_list(), orc.hb_list())
    assert rel_force_err(eng.force()[0], orc.force()[0]) < FORCE_TOL[precision]
    eng.set_noise(noise)
    orc.set_noise(noise[:, None])
    eng.time_integral_pre()
    orc.time_integral_pre()
    eng.step(4)
    eng.step(steps - 4)
    orc.step(steps)
    assert np.abs(eng.get_state()[0] - orc.get_state()[0].reshape(-1, 3)).max() < POS_TOL[precision]
    eng.close()


def ion_box():
    systems, par, _ = synth.workload_c2()
    return systems[0], dict(par, launch_ctas=1)


def test_periodic_binned_lists_bit_exact(tis_lib):
    s, par = ion_box()
    eng = Engine([s], par, [300.0])
    run = eng.launch()
    assert run["layout"] == 1 and binned(s, par, run["threads"] // 32)
    orc = Oracle(s, dict(par, precision=0), [300.0])
    eng.set_state(s["xyz"])
    orc.set_state(s["xyz"][None])
    eng.neighbor()
    orc.neighbor()
    compare_lists(eng, orc)
    assert len(eng.exv_list()) > 0
    eng.close()


def test_periodic_binned_lists_of_skin_rebuilds(tis_lib):
    """One step per call; whenever a step rebuilt the lists, they equal the
    oracle's from the positions that step started from."""
    s, par = ion_box()
    par = dict(par, n_step_neighbor=0, neigh_margin=2.0)
    eng = Engine([s], par, [300.0])
    run = eng.launch()
    assert run["layout"] == 1 and binned(s, par, run["threads"] // 32)
    eng.set_state(s["xyz"])
    eng.time_integral_pre()
    orc = Oracle(s, dict(par, precision=0), [300.0])
    checked, before = 0, eng.rebuild_info(1)[0]
    for _ in range(600):
        p0 = eng.get_pxyz()
        assert eng.step(1) >= 0
        now = eng.rebuild_info(1)[0]
        if now > before:
            orc.set_state(p0[None])
            orc.neighbor()
            compare_lists(eng, orc)
            checked += 1
            if checked == 3:
                break
        before = now
    assert checked == 3
    eng.close()
