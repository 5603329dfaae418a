"""Steps of small fields with a phase per axis: few wide planes, and more
planes than SMs, at the edges of the rule that takes them, with and without
sources and nodes, one step and several in a call (the first step's sources
are applied in another place than the later ones'), agents sharing voxels.
Against the oracle at the suite's 1e-12."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from biofvm_b200._abi import STEP_BULK, STEP_CELLS, STEP_DIFFUSION
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SHAPES = [((64, 64, 1), 1), ((64, 64, 2), 20), ((64, 47, 8), 5), ((64, 64, 9), 1),
          ((43, 43, 4), 2), ((57, 33, 1), 3), ((33, 57, 2), 7), ((41, 41, 4), 2),
          ((50, 50, 50), 4), ((33, 40, 64), 3), ((64, 16, 50), 10), ((4, 3, 60), 300)]


@pytest.mark.parametrize("shape,S", SHAPES)
@pytest.mark.parametrize("steps", [1, 3])
def test_steps_equal_the_oracle(shape, S, steps):
    scn = W.mixed_small(shape=shape, S=S, n_agents=400, seed=sum(shape) + S)
    with Solver(0) as sv:
        load_scenario(sv, scn)
        assert sv.get_grid_steps() > 0
        sv.step(scn.dt, steps)
        err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, steps, 7))
    assert np.all(err <= 1e-12), err


@pytest.mark.parametrize("flags", [STEP_DIFFUSION, STEP_DIFFUSION | STEP_BULK,
                                   STEP_DIFFUSION | STEP_CELLS])
@pytest.mark.parametrize("dirichlet", [True, False])
@pytest.mark.parametrize("shape,S", [((64, 64, 1), 2), ((50, 50, 50), 4)])
def test_parts_of_a_step(shape, S, dirichlet, flags):
    scn = W.mixed_small(shape=shape, S=S, n_agents=400, seed=9, dirichlet=dirichlet)
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.step(scn.dt, 2, flags)
        sv.step(scn.dt, 1, flags)
        err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, 3, flags))
    assert np.all(err <= 1e-12), err


def test_all_agents_in_one_voxel():
    """One voxel's 300 agents, in list order, and voxels of two and three."""
    scn = W.mixed_small(shape=(64, 64, 2), S=2, n_agents=320, seed=12)
    scn.agent_pos[:300] = scn.agent_pos[0]
    scn.agent_pos[300:310:2] = scn.agent_pos[301:311:2]
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.step(scn.dt, 3)
        err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, 3, 7))
    assert np.all(err <= 1e-12), err


def test_solvers_side_by_side():
    """Several solvers' steps on their own streams at once."""
    scns = [W.mixed_small(shape=s, S=S, n_agents=100, seed=k)
            for k, (s, S) in enumerate([((64, 64, 1), 1), ((50, 50, 50), 4), ((50, 40, 30), 2)])]
    sols = [Solver(0) for _ in scns]
    try:
        for sv, scn in zip(sols, scns):
            load_scenario(sv, scn)
        for _ in range(4):
            for sv, scn in zip(sols, scns):
                sv.step(scn.dt, 1)
        for sv, scn in zip(sols, scns):
            err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, 4, 7))
            assert np.all(err <= 1e-12), (scn.shape, err)
    finally:
        for sv in sols:
            sv.close()
