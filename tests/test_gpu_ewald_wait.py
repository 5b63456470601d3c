"""Waits for the reciprocal Ewald sum that give up (split_ewald.cuh): with a
limit of one poll the launch still takes all its steps and ends, the call
returns TIS_E_TIMEOUT, the status says so, and the GPU serves the next
context.  No fault and no endless wait is involved: a wait that runs out
raises a flag with which every wait returns at once."""
import ctypes as C

import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine, TisError

pytestmark = pytest.mark.gpu
TIS_E_TIMEOUT = -5


def box(precision):
    s = synth.set_friction(synth.dt15_chain(12, 3, stem=3), 0.5)
    s = synth.add_ions(s, 40.0, {"Mg": 2, "K": 10, "Cl": 3}, 9, clash=5.0)
    return s, synth.dt15_params(i_periodic=1, psize=(40.0, 40.0, 40.0), i_ele=2, ewld_alpha=0.2, ewld_hmax=8.0,
                                cutoff_ele=19.9, n_step_neighbor=0, precision=precision, launch_ctas=4)


@pytest.mark.parametrize("precision", [0, 1])
def test_wait_that_runs_out(tis_lib, precision):
    s, par = box(precision)
    good, bad = Engine([s], par, [300.0]), Engine([s], par, [300.0])
    hook = tis_lib.tis_test_ewald_polls
    hook.argtypes = [C.c_void_p, C.c_int32]
    for e in (good, bad):
        e.set_state(s["xyz"])
        e.time_integral_pre()
        assert e.step(5) >= 0
        assert e.status()["wait_timeout"] == 0
    assert hook(bad.h, 0) < 0
    assert hook(bad.h, 1) == 0
    launches = bad.launch_count()
    with pytest.raises(TisError) as err:
        bad.step(50)
    assert err.value.code == TIS_E_TIMEOUT
    assert bad.launch_count() - launches == 1
    assert bad.status()["wait_timeout"] == 1 and bad.status()["step"] == 55
    bad.close()
    ref = Engine([s], par, [300.0])
    ref.set_state(s["xyz"])
    ref.time_integral_pre()
    ref.step(5)
    for e in (good, ref):
        e.step(50)
    assert all(np.array_equal(a, b) for a, b in zip(good.get_state(), ref.get_state()))
    good.close()
    ref.close()
