"""Bulk lists on both sides of the rule that takes runs of voxels (96 elements a
run on average), bit for bit against the oracle."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from biofvm_b200._abi import STEP_BULK
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,length", [(1, 95), (1, 97), (4, 23), (4, 24), (4, 25), (16, 1), (16, 5),
                                      (16, 6), (20, 1), (20, 5), (32, 2), (32, 3), (33, 9)])
def test_runs_around_the_rule(S, length):
    scn = W.mixed_small(shape=(50, 40, 20), S=S, n_agents=0, seed=S + length, bulk=False,
                        dirichlet=False)
    vox = np.flatnonzero(np.arange(scn.num_voxels) % (length + 2) < length).astype(np.int64)
    rng = np.random.default_rng(length)
    table = rng.uniform(0.1, 3.0, (3, 3, S))
    row = (np.arange(vox.size) * 3) // vox.size
    scn.bulk_voxels = vox
    scn.bulk_supply, scn.bulk_target, scn.bulk_uptake = (
        np.ascontiguousarray(table[row, k]) for k in range(3))
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.step(scn.dt, 2, STEP_BULK)
        assert np.array_equal(sv.get_densities(), O.oracle_run(scn, 2, STEP_BULK))
