"""State copies through the pinned staging memory: set_state and set_step
return before the device is done, so whatever reads next must see their work,
and a second set_state must not overwrite what the first still copies."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 300])
def test_readers_see_the_last_state(tis_lib, copies):
    s = synth.set_friction(synth.dt15_chain(20, 3), 0.5)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=0)
    eng = Engine([s] * copies, par, [300.0] * copies, nrep=[1] * copies)
    rng = np.random.default_rng(1)
    base = np.vstack([s["xyz"]] * copies)
    for k in range(6):
        eng.set_state(base + 100.0)
        x = base + 0.01 * rng.normal(size=base.shape)
        v = rng.normal(size=base.shape) if k % 2 else None
        a = rng.normal(size=base.shape) if k % 3 else None
        eng.set_state(x, v, a)
        sent = x.copy()
        x[:] = np.nan                      # the call has taken its own copy
        if k % 2:
            assert np.array_equal(eng.get_pxyz(), sent)
        gx, gv, ga = eng.get_state()
        assert np.array_equal(gx, sent)
        assert np.array_equal(gv, np.zeros_like(base) if v is None else v)
        assert np.array_equal(ga, np.zeros_like(base) if a is None else a)
    eng.close()


def test_step_number_is_set_for_every_replica(tis_lib):
    s = synth.set_friction(synth.dt15_chain(12, 3), 0.5)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=0)
    eng = Engine([s] * 300, par, [300.0] * 300, nrep=[1] * 300)
    out = []
    for _ in range(2):                     # the counter-based noise follows the step number
        eng.set_step(1000)
        eng.set_state(np.vstack([s["xyz"]] * 300))
        eng.time_integral_pre()
        eng.step(3)
        assert (eng.steps() == 1003).all()
        out.append(eng.get_state())
    for p, q in zip(*out):
        assert np.array_equal(p, q)
    eng.close()
