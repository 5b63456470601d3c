"""Rows of a launch table that the caller names (tis_params.launch_table) are
followed as they are: the trajectory is bit for bit that of the same
configuration asked for by the launch fields (the order of each bead's sum,
hence its last bits, tells split replicas from the others), and a row without a number of
CTAs leaves the choice to the library."""
import numpy as np
import pytest

from tis_b200 import autotune, synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu

ONE = dict(launch_threads=256, launch_group=4, launch_ctas=1, launch_noise_sweep=1, launch_order=1, launch_sweep=2)
PAIR = dict(launch_threads=512, launch_group=4, launch_ctas=2, launch_noise_sweep=1, launch_order=1, launch_sweep=1)
ZERO = {k: 0 for k in ONE}


def moved(s, par, temps):
    eng = Engine([s], par, temps)
    eng.set_state(np.tile(s["xyz"], (len(temps), 1)))
    eng.time_integral_pre()
    eng.step(60)
    out = eng.get_state()
    eng.close()
    return out


@pytest.mark.parametrize("precision,cfg,other", [
    (0, ONE, ZERO), (1, ONE, ZERO), (1, PAIR, ZERO), (0, dict(ZERO, launch_ctas=8), ONE), (1, ZERO, ONE)])
def test_row_of_a_named_table_is_followed(tis_lib, tmp_path, precision, cfg, other):
    s = synth.set_friction(synth.dt15_chain(60, 4, hb_fraction=0.3), 0.5)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=precision)
    temps = [290.0, 310.0]
    key = autotune.workload_key([s], par, [2])
    table = tmp_path / "t.tsv"
    autotune.merge_rows(str(table), {key: autotune.format_row(key, cfg, 1.0)})
    got = moved(s, dict(par, launch_table=str(table)), temps)
    same = moved(s, dict(par, launch_table="", **cfg), temps)
    assert all(np.array_equal(a, b) for a, b in zip(got, same))
    assert not all(np.array_equal(a, b) for a, b in zip(got, moved(s, dict(par, launch_table="", **other), temps)))


def test_tuner_measures_the_split_and_the_librarys_choice(tis_lib):
    s = synth.set_friction(synth.dt15_chain(60, 4, hb_fraction=0.3), 0.5)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=1)
    cfgs = autotune.candidates([s], par, [1])
    assert {c["launch_ctas"] for c in cfgs} == {0, 1, 2, 4, 8, 16}
    for c in cfgs[:4]:
        assert autotune.time_config([s], par, [300.0], [1], c, steps=20, reps=1) > 0
