"""An Ewald ladder held by one context and by two ranks' shares (in one
process: their kernels never wait on each other).  Whether the reciprocal sum
runs beside the split lanes or in kernels of its own is decided for the whole
ladder, so every replica moves bit-identically in either layout: on both
sides of the limit (26 replicas of 4 CTAs leave no room, their halves would;
12 leave room)."""
import numpy as np
import pytest

from tis_b200 import remd, synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu


def box():
    s = synth.set_friction(synth.dt15_chain(12, 3, stem=3), 0.5)
    s = synth.add_ions(s, 40.0, {"Mg": 2, "K": 10, "Cl": 3}, 9, clash=5.0)
    return s, synth.dt15_params(i_periodic=1, psize=(40.0, 40.0, 40.0), i_ele=2, ewld_alpha=0.2, ewld_hmax=8.0,
                                cutoff_ele=19.9, n_step_neighbor=0)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nall", [12, 26])
def test_ewald_ladder_contexts_match_one_context(tis_lib, nall, precision):
    s, par = box()
    par = dict(par, precision=precision, launch_ctas=4)
    n, ladder = s["nmp"], synth.temperature_ladder(nall, 280.0, 400.0)
    engines = [(1, Engine([s], par, ladder, nrep=[nall]))]
    for rank in range(2):
        first, count = remd.ladder_share(nall, 2, rank)
        engines.append((first, Engine([s], par, ladder[first - 1:first - 1 + count], nrep=[count],
                                      ladder=(ladder, first))))
    launches = []
    for _, e in engines:
        e.set_state(np.tile(s["xyz"], (e.nlane, 1)))
        e.time_integral_pre()
        l0 = e.launch_count()
        e.step(20)
        launches.append(e.launch_count() - l0)
    assert (launches[0] == 1) == (nall == 12)
    x1, v1, _ = engines[0][1].get_state()
    for first, e in engines[1:]:
        x, v, _ = e.get_state()
        part = slice((first - 1) * n, (first - 1 + e.nlane) * n)
        assert np.array_equal(x, x1[part]) and np.array_equal(v, v1[part])
    for _, e in engines:
        e.close()
