"""Charged rows of split replicas whose partner lists do not fit the shared
memory read the bits of the row instead, in the order of the list, so a
replica's forces and trajectory do not depend on the number of CTAs, bit for
bit: Debye-Hueckel rows of 32 threads and Ewald rows of 8, with lists
(more CTAs) and without (fewer)."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu


def system(kind):
    if kind == "ewald":
        systems, par, _ = synth.workload_c2()
        return systems[0], dict(par, cutoff_ele=70.0, n_step_neighbor=0)
    s = synth.set_friction(synth.dt15_chain(int(kind), 70 + int(kind), hb_fraction=0.3), 0.5)
    return s, synth.dt15_params(ionic_strength=0.05, n_step_neighbor=0)


@pytest.mark.parametrize("kind,precision,few,many", [
    ("400", 1, 8, 16), ("280", 1, 4, 16), ("240", 0, 4, 16), ("ewald", 1, 4, 16), ("ewald", 0, 8, 16)])
def test_bits_and_lists_add_alike(tis_lib, kind, precision, few, many):
    s, par = system(kind)
    out, lists = [], []
    for ctas in (few, many):
        eng = Engine([s], dict(par, precision=precision, launch_ctas=ctas), [300.0])
        eng.set_state(s["xyz"])
        eng.time_integral_pre()
        f = eng.force()[0]
        eng.step(12)
        out.append((f,) + eng.get_state())
        lists.append(eng.launch()["row_lists"])
        eng.close()
    assert lists == [0, 1]
    for a, b in zip(*out):
        assert np.array_equal(a, b)
