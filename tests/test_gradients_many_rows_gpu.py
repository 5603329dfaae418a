"""compute_all_gradient_vectors bit for bit against the oracle on both sides of
the rule that takes four rows at a time (27 blocks of a row an SM, four rows a
plane): rows that do and do not fill a warp's elements, row counts that are and
are not multiples of four, extreme values, FP32 fields."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def gradients(scn, p, precision):
    with Solver(0) as sv:
        load_scenario(sv, scn)
        if precision != 64:
            sv.set_precision(precision)
        sv.set_densities(p)
        sv.compute_all_gradient_vectors()
        return sv.get_gradient_vectors(), sv.get_densities()


@pytest.mark.parametrize("shape,S", [((16, 64, 62), 1), ((16, 64, 63), 1), ((33, 66, 64), 1),
                                     ((40, 71, 60), 2), ((300, 45, 50), 1), ((17, 65, 64), 5),
                                     ((5, 3, 1400), 2), ((5, 4, 1100), 2), ((1, 2500, 2), 3),
                                     ((3, 4001, 1), 1)])
@pytest.mark.parametrize("dx", [10.0, 3.3])
def test_many_rows(shape, S, dx):
    scn = W.mixed_small(shape=shape, S=S, n_agents=0, seed=sum(shape) + S, dx=dx, dirichlet=False,
                        bulk=False)
    for precision in (64, 32):
        g, p = gradients(scn, scn.p0, precision)
        assert np.array_equal(g, O.oracle_gradients(p, scn.shape, scn.mesh.dx))


@pytest.mark.parametrize("shape", [(40, 12, 6), (20, 70, 60)])
def test_extreme_values(shape):
    scn = W.mixed_small(shape=shape, S=2, n_agents=0, seed=3, dirichlet=False, bulk=False)
    rng = np.random.default_rng(4)
    p = scn.p0.copy()
    at = rng.permutation(p.size)[:2000]
    p.ravel()[at] = rng.choice([0.0, -0.0, 1e300, -1e300, 1e-310, 5e-324, np.inf, -np.inf,
                                2.0 ** -900, 1.7e308], 2000)
    p[:200] = 0.25  # equal neighbours: zero differences
    with np.errstate(all="ignore"):
        g, q = gradients(scn, p, 64)
        assert np.array_equal(g, O.oracle_gradients(q, scn.shape, scn.mesh.dx), equal_nan=True)
