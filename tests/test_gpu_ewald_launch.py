"""The reciprocal Ewald sum beside the split lanes, all steps in one launch
(split_ewald.cuh), against the CPU restatement and against the separate
kernels a batch takes that leaves no CTAs for it.

Sizes: 4, 8 and 16 CTAs per replica (256 and 512 threads: whole and half
columns), columns of 1 to 9 and of 1 to 11 vectors, one replica and several
(fewer charges than workers and more).  Tolerances as in the trajectory test
of the separate kernels: FP64 1e-8 A, mixed 1e-4 A."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from tis_b200 import synth
from tis_b200.engine import Engine

pytestmark = pytest.mark.gpu

TOL = {0: 1e-8, 1: 1e-4}


def box(hmax):
    s = synth.set_friction(synth.dt15_chain(12, 3, stem=3), 0.5)
    s = synth.add_ions(s, 40.0, {"Mg": 2, "K": 10, "Cl": 3}, 9, clash=5.0)
    par = synth.dt15_params(i_periodic=1, psize=(40.0, 40.0, 40.0), i_ele=2, ewld_alpha=0.2, ewld_hmax=hmax,
                            cutoff_ele=19.9)
    return s, par


def ion_box():
    systems, par, _ = synth.workload_c2()
    return systems[0], par


@pytest.mark.parametrize("name,precision,ctas,copies", [
    ("h8", 0, 4, 1), ("h8", 0, 4, 3), ("h8", 1, 8, 2), ("h11", 0, 8, 1), ("h11", 1, 4, 1),
    ("c2", 0, 16, 1), ("c2", 1, 16, 2), ("c2", 1, 8, 1)])
def test_trajectory_against_oracle(tis_lib, name, precision, ctas, copies):
    s, par = ion_box() if name == "c2" else box({"h8": 8.0, "h11": 11.0}[name])
    par = dict(par, precision=precision, n_step_neighbor=0, launch_ctas=ctas)
    eng = Engine([s] * copies, par, [300.0] * copies, nrep=[1] * copies)
    rng = np.random.default_rng(11)
    noise = rng.normal(size=(7, eng.nbead, 3))
    start = [s["xyz"] + 0.01 * rng.normal(size=s["xyz"].shape) for _ in range(copies)]
    eng.set_state(np.vstack(start))
    eng.set_noise(noise)
    eng.time_integral_pre()
    eng.step(4)
    eng.step(2)
    x = eng.get_state()[0]
    eng.close()
    n = s["nmp"]
    for k in range(copies):
        orc = Oracle(s, dict(par, precision=0), [300.0])
        orc.set_state(start[k][None])
        orc.set_noise(noise[:, k * n:(k + 1) * n].reshape(7, 1, n, 3))
        orc.time_integral_pre()
        orc.step(6)
        assert np.abs(x[k * n:(k + 1) * n] - orc.get_state()[0].reshape(-1, 3)).max() < TOL[precision], k
        orc.close()


def test_batch_without_room_takes_the_separate_kernels(tis_lib):
    """60 replicas of 4 CTAs leave no room for workers; the first moves as it
    does alone, to the rounding of sums taken in another order."""
    s, par = box(8.0)
    par = dict(par, precision=0, n_step_neighbor=0, launch_ctas=4)
    out = []
    for copies in (1, 60):
        eng = Engine([s] * copies, par, [300.0] * copies, nrep=[1] * copies)
        noise = np.random.default_rng(5).normal(size=(7, s["nmp"], 3))
        eng.set_noise(np.tile(noise, (1, copies, 1)))
        eng.set_state(np.vstack([s["xyz"]] * copies))
        eng.time_integral_pre()
        l0 = eng.launch_count()
        eng.step(6)
        out.append((eng.get_state()[0][:s["nmp"]], eng.launch_count() - l0))
        eng.close()
    assert out[0][1] == 1 and out[1][1] > 6
    assert np.abs(out[0][0] - out[1][0]).max() < TOL[0]
