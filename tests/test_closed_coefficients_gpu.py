"""Coefficients that do not have the closed form (negative diffusion, a decay
rate of -3 / dt or below, one such density among ordinary ones) are solved by
elimination, as the reference solves them; a growth rate above -3 / dt has the
closed form.  Against the oracle, whose elimination agrees with a dense solve
to 1e-15 on these systems.

Bars: the suite's 1e-12 where the lines are diagonally dominant; the
indefinite lines (c1 = -0.3, condition numbers 39, 10 and 12 along x, y, z)
may lose their product, 4.7e3, times a few roundings each: 1e-10."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def scenario(shape, c1, c2, dims=3):
    scn = W.mixed_small(shape=shape, S=len(c1), n_agents=40, seed=sum(shape), bulk=True)
    scn.D = np.array(c1) * scn.mesh.dx ** 2 / scn.dt
    scn.decay = np.array(c2) * dims / scn.dt
    return scn


CASES = {
    "growth_past_one_step": ((40, 33, 70), (0.1, 0.05), (-2.0, -2.0), 1e-12),
    "one_density_of_three": ((24, 20, 16), (1.0, 0.1, 3.0), (0.01, -2.0, 0.02), 1e-12),
    "growth": ((40, 33, 70), (5.0, 0.5), (-0.5, -0.25), 1e-12),
    "negative_diffusion": ((24, 20, 16), (-0.2, 1.0), (0.0, 0.1), 1e-12),
    "indefinite": ((7, 6, 5), (-0.3, -0.15), (0.0, 0.0), 1e-10),
}


@pytest.mark.parametrize("grid", [True, False], ids=["grid_steps", "sweeps"])
@pytest.mark.parametrize("name", CASES)
def test_unusual_coefficients(name, grid):
    shape, c1, c2, tol = CASES[name]
    scn = scenario(shape, c1, c2)
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.set_grid_steps(grid)
        sv.step(scn.dt, 2)
        err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, 2, 7))
    assert np.all(err <= tol), err


def test_unusual_coefficients_in_2d():
    scn = scenario((70, 33, 1), (0.1, 1.0), (-2.0, 0.1), dims=2)
    scn.bulk_voxels, scn.agent_pos = None, None
    with Solver(0) as sv:
        load_scenario(sv, scn)
        for _ in range(2):
            sv.simulate_diffusion_decay_2d(scn.dt)
        err = O.max_rel_err(sv.get_densities(), O.oracle_lod2d_run(scn, 2))
    assert np.all(err <= 1e-12), err


def test_a_new_setup_follows_its_coefficients():
    """Ordinary coefficients, then ones without the closed form, then ordinary
    ones again, with a reset of the setup between."""
    scn = scenario((24, 20, 16), (1.0, 0.3), (0.01, 0.02))
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.set_grid_steps(False)
        for c1, c2 in (((1.0, 0.3), (0.01, 0.02)), ((0.1, 0.05), (-2.0, -2.0)),
                       ((2.0, 0.3), (0.01, 0.02))):
            step = scenario((24, 20, 16), c1, c2)
            step.p0 = sv.get_densities()
            sv.set_coefficients(step.D, step.decay)
            sv.reset_diffusion_setup()
            sv.step(scn.dt, 1)
            err = O.max_rel_err(sv.get_densities(), O.oracle_run(step, 1, 7))
            assert np.all(err <= 1e-12), (c1, c2, err)
