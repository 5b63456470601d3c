"""States larger than the pinned staging memory (1 MB) go through its two
halves part by part: values, orders of calls, missing arrays and sizes around
the limits (whole state, a part's remainder of one bead, many parts)."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,copies", [(20, 240), (20, 250), (20, 368), (27, 256), (100, 150)])
def test_large_states(tis_lib, nt, copies):
    s = synth.set_friction(synth.dt15_chain(nt, 3), 0.5)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=0)
    eng = Engine([s] * copies, par, [300.0] * copies, nrep=[1] * copies)
    rng = np.random.default_rng(nt + copies)
    base = np.vstack([s["xyz"]] * copies)
    for k in range(5):
        eng.set_state(base + 100.0, base)
        x = base + 0.01 * rng.normal(size=base.shape)
        v = rng.normal(size=base.shape) if k % 2 else None
        a = rng.normal(size=base.shape) if k % 3 else None
        eng.set_state(x, v, a)
        sent = x.copy()
        x[:] = np.nan                      # the call has taken its own copy
        if k == 3:
            assert np.array_equal(eng.get_pxyz(), sent)
        gx, gv, ga = eng.get_state()
        assert np.array_equal(gx, sent)
        assert np.array_equal(gv, np.zeros_like(base) if v is None else v)
        assert np.array_equal(ga, np.zeros_like(base) if a is None else a)
    out = []
    for _ in range(2):                     # and through a step
        eng.set_step(0)
        eng.set_state(base, base * 0.01)
        eng.time_integral_pre()
        eng.step(2)
        out.append(eng.get_state())
    assert all(np.array_equal(p, q) for p, q in zip(*out)) and np.isfinite(out[0][0]).all()
    eng.close()
