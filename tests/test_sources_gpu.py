"""The stand-alone bulk kernel over runs of voxels that share a rate row, bit
for bit against the oracle: runs of every length around what a warp takes,
several rows, densities that fill and do not fill a warp, scattered voxels
(which keep the per-voxel kernel), extreme values, FP32 fields."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from biofvm_b200._abi import STEP_BULK
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def bulk_scenario(S, pieces, rows, seed):
    rng = np.random.default_rng(seed)
    scn = W.mixed_small(shape=(61, 30, 12), S=S, n_agents=0, seed=seed, bulk=False,
                        dirichlet=False)
    vox, row = [], []
    at = 3
    for n in pieces:
        vox += range(at, at + n)
        row += [int(rng.integers(rows))] * n
        at += n + int(rng.integers(0, 2))  # some runs touch the next one
    table = rng.uniform(0.1, 3.0, (rows, 3, S))
    scn.bulk_voxels = np.array(vox, np.int64)
    scn.bulk_supply, scn.bulk_target, scn.bulk_uptake = (
        np.ascontiguousarray(table[row, k]) for k in range(3))
    return scn


@pytest.mark.parametrize("S", [1, 2, 3, 5, 8, 10, 16, 31, 32, 33])
def test_bulk_runs_equal_the_oracle(S):
    most = max(1, 32 // S * 8)
    pieces = [1, 2, most - 1, most, most + 1, 2 * most, 3 * most + 5, 40, 7]
    scn = bulk_scenario(S, [max(1, n) for n in pieces] * 3, rows=4, seed=S)
    scn.p0.ravel()[::97] = np.resize([0.0, 1e300, -1e-300, 5e-324, -0.0], scn.p0.size // 97 + 1)[
        :len(scn.p0.ravel()[::97])]
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.step(scn.dt, 3, STEP_BULK)
        assert np.array_equal(sv.get_densities(), O.oracle_run(scn, 3, STEP_BULK))


@pytest.mark.parametrize("pieces", [[1] * 300, [500, 500]], ids=["scattered", "long"])
def test_bulk_on_an_fp32_field(pieces):
    scn = bulk_scenario(4, pieces, rows=3, seed=9)
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.set_precision(32)
        sv.set_densities(scn.initial_field())
        sv.step(scn.dt, 1, STEP_BULK)
        got = sv.get_densities()
    scn.p0 = scn.p0.astype(np.float32).astype(np.float64)
    ref = O.oracle_run(scn, 1, STEP_BULK).astype(np.float32).astype(np.float64)
    assert np.array_equal(got, ref)
