"""Mixed precision, split replicas: whether a tertiary stack turns secondary
stacks off (force_dtrna_stack_nlocal.F90:83-92, closer than 10 A to its
native distance) is decided in FP64 from the FP64 positions, as the reference
decides it, also 2,000 A from the origin, where FP32 hi and lo parts carry a
coordinate to 4e-12 A only.  The native distance is set 2e-13 to 2e-12 A to
either side of the limit; the forces must be the oracle's for this side, not
those for the other one (their difference, 0.07 kcal/mol/A, is far above the
FP32 rounding)."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def oracle_force(s, par, x):
    orc = Oracle(s, dict(par, precision=0), [300.0])
    orc.set_state(x[None])
    orc.neighbor()
    f = orc.force()[0]
    orc.close()
    return f


@pytest.mark.parametrize("ctas", [4, 8])
@pytest.mark.parametrize("offset", [0.0, 1950.0])
def test_exclusion_is_the_references(tis_lib, ctas, offset):
    base = synth.hairpin_tertiary()
    rng = np.random.default_rng(4)
    par = synth.dt15_params(ionic_strength=0.15, n_step_neighbor=0, precision=1)
    decided = set()
    for trial in range(12):
        s = dict(base)
        x = base["xyz"] + rng.normal(0.0, 0.02, size=base["xyz"].shape) + offset * np.array([1.0, -0.9, 0.8])
        m = np.asarray(s["idtrna_tst2mp"]).reshape(-1, 6)[2] - 1
        v = x[m[0]] - x[m[1]]
        dist = np.sqrt((v[0] * v[0] + v[1] * v[1]) + v[2] * v[2])
        nat = np.array(s["dtrna_tst_nat"], dtype=np.float64).reshape(-1, 6).copy()
        side = (1.0 if trial % 2 else -1.0) * rng.uniform(2.0e-13, 2.0e-12)
        other = nat.copy()
        nat[2, 0], other[2, 0] = dist - 10.0 + side, dist - 10.0 - side
        ref, wrong = (oracle_force(dict(s, dtrna_tst_nat=n), par, x) for n in (nat, other))
        decided.add(bool(dist - nat[2, 0] < 10.0))
        assert np.abs(ref - wrong).max() > 0.01
        eng = Engine([dict(s, dtrna_tst_nat=nat)], dict(par, launch_ctas=ctas), [300.0])
        eng.set_state(x)
        eng.neighbor()
        f = eng.force()[0]
        eng.close()
        share = ((f - ref) * (wrong - ref)).sum() / ((wrong - ref) ** 2).sum()   # 0: the right one, 1: the other
        assert abs(share) < 0.5, (trial, share)
    assert decided == {True, False}
