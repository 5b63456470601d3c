"""What each replica's steps run on (tis_get_launch), so that tests of the
library's own choices see which kernel ran: the layouts that a caller asks
for, a batch whose long chains are split beside short ones, charged rows with
and without partner lists, and status fields that describe the launch in
use."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu


def chain(n):
    return synth.set_friction(synth.dt15_chain(n, 70 + n, hb_fraction=0.3), 0.5)


@pytest.mark.parametrize("cfg,precision,want", [
    (dict(launch_ctas=1), 1, (1, 1, 256)), (dict(launch_ctas=1, launch_threads=128), 0, (1, 1, 128)),
    (dict(launch_ctas=2), 1, (2, 2, 512)), (dict(launch_ctas=4), 0, (3, 4, 256)),
    (dict(launch_ctas=8), 1, (3, 8, 256)), (dict(launch_ctas=16), 1, (3, 16, 256))])
def test_layout_that_was_asked_for(tis_lib, cfg, precision, want):
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=precision)
    cfg = dict(cfg, launch_threads=256) if "launch_threads" not in cfg else cfg
    eng = Engine([chain(33)], dict(par, **cfg), [300.0] * 2)
    for irep in (1, 2):
        assert tuple(eng.launch(irep)[k] for k in ("layout", "ctas", "threads")) == want
    st = eng.status()
    assert st["launch_source"] == 2 and st["threads_per_cta"] == want[2]
    assert st["ctas_per_lane"] == (2 if want[0] == 2 else 1)
    with pytest.raises(RuntimeError):
        eng.launch(3)
    eng.close()


def test_single_replica_is_split_and_says_so(tis_lib):
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=1)
    eng = Engine([chain(200)], par, [300.0])
    run, st = eng.launch(), eng.status()
    assert run["layout"] == 3 and run["ctas"] >= 4 and run["row_lists"] == 1
    assert (st["launch_source"], st["threads_per_cta"], st["group"], st["sweep"]) == (0, run["threads"], 8, 2)
    eng.close()


def test_long_chains_of_a_batch_are_split_beside_short_ones(tis_lib):
    """The batch of test_batch_with_some_lanes_split: both kernels run, as two
    launches of one step call."""
    systems = [chain(k) for k in [300] * 12 + [20] * 150]
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=0)
    eng = Engine(systems, par, [300.0] * len(systems), nrep=[1] * len(systems))
    layout = [eng.launch(k + 1)["layout"] for k in range(len(systems))]
    assert layout == [3] * 12 + [1] * 150
    eng.set_state(np.vstack([s["xyz"] for s in systems]))
    eng.time_integral_pre()
    before = eng.launch_count()
    eng.step(3)
    assert eng.launch_count() - before == 2
    eng.close()


@pytest.mark.parametrize("ctas,fits", [(8, 0), (16, 1)])
def test_partner_lists_of_long_rows(tis_lib, ctas, fits):
    s = chain(400)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=1, launch_ctas=ctas)
    eng = Engine([s], par, [300.0])
    eng.set_state(s["xyz"])
    eng.neighbor()
    eng.force()
    run = eng.launch()
    assert (run["layout"], run["ctas"], run["row_lists"]) == (3, ctas, fits)
    eng.close()


def test_ladder_with_long_cadence_is_split_over_two_ctas(tis_lib):
    s = synth.set_friction(synth.dt15_chain(76, 5), 0.5)
    for every, want in ((0, (3, 2)), (10, (2, 2))):
        par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=every, precision=1)
        eng = Engine([s], par, list(np.geomspace(280.0, 400.0, 64)))
        assert all((eng.launch(k)["layout"], eng.launch(k)["ctas"]) == want for k in (1, 64))
        eng.close()


def test_brownian_hi_has_no_lane_kernel(tis_lib):
    eng = Engine([synth.bead_chain(24, 7)], synth.bdhi_params(), [300.0])
    assert eng.launch() == dict(layout=0, ctas=0, threads=0, row_lists=0)
    eng.close()


def test_a_recorded_period_of_a_batch_with_both_kernels(tis_lib):
    """tis_run records the two kernels' launches on two streams: the same
    steps as tis_step, bit for bit, also when replayed."""
    systems = [chain(k) for k in [300] * 12 + [20] * 150]
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=0)
    out = []
    for recorded in (False, True):
        eng = Engine(systems, par, [300.0] * len(systems), nrep=[1] * len(systems))
        assert eng.launch(1)["layout"] == 3 and eng.launch(162)["layout"] == 1
        eng.set_state(np.vstack([s["xyz"] for s in systems]))
        eng.time_integral_pre()
        for _ in range(2):
            if recorded:
                eng.run(2, 4, exchange=False)
            else:
                eng.step(8)
        out.append(eng.get_state())
        eng.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))
