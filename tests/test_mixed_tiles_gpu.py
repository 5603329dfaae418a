"""FP32 fields in FP64 arithmetic on the TMA-fed line kernel, whose tile rows
are then 64 bytes: odd numbers of points, around the tensor boxes' 256, with
strides that are multiples of 16 bytes (others take the direct kernel).
Against the oracle at the suite's 1e-6 for such fields; the tuner, which times
that kernel, leaves the field as it was."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from biofvm_b200._abi import FP32_FP64MATH, PATH_TMA
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def mixed(scn):
    sv = Solver(0)
    load_scenario(sv, scn)
    sv.set_precision(FP32_FP64MATH)
    sv.set_densities(scn.initial_field())
    return sv


@pytest.mark.parametrize("n", [1, 3, 5, 33, 127, 255, 256, 257, 511, 513])
def test_odd_lines(n):
    for shape in ((12, n, 5), (12, 5, n)):
        scn = W.mixed_small(shape=shape, S=2, n_agents=60, seed=n)
        with mixed(scn) as sv:
            sv.set_kernel_path(PATH_TMA)
            sv.step(scn.dt, 2)
            err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, 2, 7))
        assert np.all(err <= 1e-6), (shape, err)


def test_the_tuner_on_odd_lines():
    scn = W.mixed_small(shape=(16, 21, 35), S=4, n_agents=60, seed=6)
    with mixed(scn) as sv:
        before = sv.get_densities()
        sv.tune_sweeps(scn.dt, 1)
        assert np.array_equal(sv.get_densities(), before)
        sv.step(scn.dt, 2)
        err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, 2, 7))
    assert np.all(err <= 1e-6), err
