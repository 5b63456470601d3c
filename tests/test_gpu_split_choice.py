"""The library's choice between one CTA, pairs of CTAs and splits counts the
list rebuilds and the launch that would run otherwise: replicas whose lists
are rebuilt every few steps keep the kernel that tests each pair once where
the split was measured slower (599 beads x 64 and a rebuild every 10 steps:
55 against 47 us a step; 899 beads 143 against 90; every 50 steps 92 against
82; 1,199 beads without electrostatics 152 against 125), and are split where
that is faster."""
import numpy as np
import pytest

from tis_b200 import remd, synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu


def layouts(nt, nlane, par, ladder=None):
    s = synth.set_friction(synth.dt15_chain(nt, 1, hb_fraction=0.3), 0.5)
    temps = list(np.linspace(290.0, 310.0, nlane))
    if ladder:
        first, count = ladder
        eng = Engine([s], par, temps[first - 1:first - 1 + count], nrep=[count], ladder=(temps, first))
    else:
        eng = Engine([s], par, temps, nrep=[nlane])
    out = {(eng.launch(k + 1)["layout"], eng.launch(k + 1)["ctas"]) for k in range(eng.nlane)}
    eng.close()
    assert len(out) == 1
    return out.pop()


@pytest.mark.parametrize("nt,nlane,every,want", [
    (200, 64, 5, (2, 2)), (200, 64, 10, (2, 2)), (300, 64, 10, (2, 2)), (300, 64, 50, (2, 2)),
    (200, 64, 0, (3, 4)), (76, 64, 0, (3, 2)), (30, 64, 10, (3, 2)), (200, 1, 10, (3, 16)), (400, 8, 0, (3, 16))])
def test_debye_hueckel_mixed(tis_lib, nt, nlane, every, want):
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=every, precision=1)
    assert layouts(nt, nlane, par) == want


def test_without_electrostatics(tis_lib):
    par = synth.dt15_params(i_ele=0, n_step_neighbor=10, precision=1)
    assert layouts(400, 64, par) == (1, 1)


def test_a_ladders_ranks_choose_alike(tis_lib):
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=10, precision=1)
    whole = layouts(200, 40, par)
    for rank in range(4):
        assert layouts(200, 40, par, ladder=remd.ladder_share(40, 4, rank)) == whole
