"""Closed-form sweeps of short lines: 8-point chunks up to 8 points and from 17
to 24, 16-point chunks between and beyond, with few columns and with enough of
them for wider blocks, nodes along x and y, in every precision mode; and lines
past 512 points of FP32 fields as tiles of 16 columns, at odd numbers of points.
Against the oracle at the suite's bars."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from biofvm_b200._abi import FP32, FP32_FP64MATH, FP64
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = {FP64: 1e-12, FP32_FP64MATH: 1e-6, FP32: 1e-5}
MODES = pytest.mark.parametrize("precision", list(TOL), ids=["fp64", "mixed", "fp32"])


def check(scn, precision):
    with Solver(0) as sv:
        load_scenario(sv, scn)
        if precision != FP64:
            sv.set_precision(precision)
            sv.set_densities(scn.initial_field())
        sv.set_grid_steps(False)
        sv.step(scn.dt, 2)
        err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, 2, 7))
    assert np.all(err <= TOL[precision]), (scn.shape, err)


@MODES
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 23, 24, 25])
def test_short_lines(n, precision):
    for shape, S in (((n, 6, 5), 3), ((4, n, 5), 2), ((5, 4, n), 1), ((n, 200, 190), 1),
                     ((200, n, 190), 1), ((200, 190, n), 1)):
        check(W.mixed_small(shape=shape, S=S, n_agents=0, seed=n + S, bulk=False), precision)


@MODES
@pytest.mark.parametrize("n", [513, 519, 520, 701, 1023])
def test_long_lines_as_tiles(n, precision):
    for shape in ((8, n, 3), (8, 3, n)):
        check(W.mixed_small(shape=shape, S=5, n_agents=0, seed=n, bulk=False), precision)
