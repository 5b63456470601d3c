"""Bond lengths of split replicas in FP64.  Coordinates on a coarse grid make
the squared length exact, and a native length within 1e-6 of the true one
makes the force show the length's own error: at most half an ulp, as a
correctly rounded square root has (a tenth more for the rounding of the
force's products)."""
import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 4, 16])
def test_bond_length_is_correctly_rounded(tis_lib, ctas):
    rng = np.random.default_rng(3)
    s = dict(synth.dt15_chain(134, 3))
    n = s["nmp"] - s["nmp"] % 2
    x = np.zeros((s["nmp"], 3))
    x[:, 0] = 20.0 * np.arange(s["nmp"])                          # pairs far apart from one another
    x[1:n:2] = x[0:n:2] + rng.integers(2048, 8192, size=(n // 2, 3)) / 2048.0
    for key in ("nba", "nst", "nhb", "nhbsite"):
        s[key] = 0
    pairs = np.arange(n).reshape(-1, 2)
    v = x[pairs[:, 1]] - x[pairs[:, 0]]
    d = np.sqrt((v.astype(np.longdouble) ** 2).sum(axis=1))
    k = 64.0
    s.update(nbd=len(pairs), ibd2mp=(pairs + 1).astype(np.int32), bd_nat=np.float64(d) * (1.0 + 1.0e-6),
             coef_bd=np.full(len(pairs), k), exv_epsilon=np.zeros(s["nmp"]), xyz=x)
    eng = Engine([s], synth.dt15_params(i_ele=0, precision=0, launch_ctas=ctas), [300.0])
    eng.set_state(x)
    eng.neighbor()
    f = eng.force()[0]
    eng.close()
    # the force on the second bead: -2 k (d - nat) v / d
    got = (f[pairs[:, 1]].astype(np.longdouble) * v).sum(axis=1) / d / (-2.0 * k) + s["bd_nat"]
    assert np.abs(f).max() > 0.0
    assert np.max(np.abs(got - d) / np.spacing(np.float64(d))) <= 0.55
