"""The Cholesky pivots' reciprocal (bdhi_kernel.cu pivot_rcp: two Newton-
Raphson steps from the instruction's approximation) against CUDA's correctly
rounded one, and factors whose pivots leave its range (subnormal, or with
subnormal reciprocals) against the restatement: no NaN, no false alarm.  1 ulp:
half an ulp of the last step's rounding, and its increment, of a relative size
of 2^-40 at most, is itself rounded.  Factors 1e-12 of the largest element, as
for ordinary pivots."""
import ctypes as C

import numpy as np
import pytest

from tis_b200 import synth
from tis_b200.engine import Engine
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def test_reciprocal_against_cuda(tis_lib):
    rng = np.random.default_rng(5)
    p = np.ldexp(rng.uniform(1.0, 2.0, size=400000), rng.integers(-1021, 1021, size=400000))
    edge = np.concatenate([np.ldexp(1.0 + np.arange(64) * 2.0 ** -52, e) for e in (-1021, -3, 0, 7, 1020)])
    p = np.ascontiguousarray(np.concatenate([p, edge, np.nextafter(edge[edge > 1.0], 0.0)]))
    own, cuda = np.empty_like(p), np.empty_like(p)
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    assert tis_lib.tis_test_pivot_rcp(ptr(p), len(p), ptr(own), ptr(cuda)) == 0
    assert np.array_equal(cuda, 1.0 / p)
    assert np.max(np.abs(own - cuda) / np.spacing(cuda)) <= 1.0


@pytest.mark.parametrize("scale", [1.0, 3.4e305, 1.5e-310])
@pytest.mark.parametrize("n", [24, 60])
def test_factor_with_extreme_pivots(tis_lib, n, scale):
    s = synth.bead_chain(n, 7)
    base = synth.bdhi_params()
    par = dict(base, viscosity=base["viscosity"] * scale)
    eng = Engine([s], par, [300.0])
    eng.set_state(s["xyz"])
    eng.set_noise(np.zeros((2, n, 3)))
    eng.time_integral_pre()
    assert eng.step(1) >= 0
    D, L = eng.hydro_tensors()
    orc = Oracle(s, par, [300.0])
    orc.set_state(s["xyz"][None])
    Dr, Lr, rc = orc.hydro_tensors()
    assert rc == 0 and np.isfinite(Lr).all() and eng.status()["not_spd"] == 0
    assert scale == 1.0 or not 1e-300 < Dr.max() < 1e300
    assert np.abs(D - Dr).max() <= 1e-12 * np.abs(Dr).max()
    assert np.isfinite(L).all() and np.abs(L - Lr).max() <= 1e-12 * np.abs(Lr).max()
    eng.close()
