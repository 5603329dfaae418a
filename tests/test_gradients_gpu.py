"""compute_all_gradient_vectors bit for bit against the oracle: rows that do
and do not fill a warp's 32 elements and 16-byte runs, row counts around the
kernel's four, axes without neighbours, and differences outside the range of
its division by a fixed divisor."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def gradients(scn, p, precision=64):
    with Solver(0) as sv:
        load_scenario(sv, scn)
        if precision != 64:
            sv.set_precision(precision)
        sv.set_densities(p)
        sv.compute_all_gradient_vectors()
        return sv.get_gradient_vectors(), sv.get_densities()


@pytest.mark.parametrize("shape,S", [((40, 12, 6), 2), ((33, 9, 5), 1), ((64, 4, 3), 4),
                                     ((300, 5, 4), 1), ((17, 13, 3), 5), ((1, 6, 5), 3),
                                     ((90, 1, 4), 2), ((70, 7, 1), 1), ((3, 3, 3), 40)])
@pytest.mark.parametrize("dx", [10.0, 3.3])
def test_gradients_equal_the_oracle(shape, S, dx):
    scn = W.mixed_small(shape=shape, S=S, n_agents=0, seed=sum(shape) + S, dx=dx, dirichlet=False,
                        bulk=False)
    for precision in (64, 32):
        g, p = gradients(scn, scn.p0, precision)
        assert np.array_equal(g, O.oracle_gradients(p, scn.shape, scn.mesh.dx))


def test_gradients_of_extreme_values():
    scn = W.mixed_small(shape=(40, 12, 6), S=2, n_agents=0, seed=3, dirichlet=False, bulk=False)
    rng = np.random.default_rng(4)
    p = scn.p0.copy()
    at = rng.permutation(p.size)[:400]
    p.ravel()[at] = rng.choice([0.0, -0.0, 1e300, -1e300, 1e-310, 5e-324, np.inf, -np.inf,
                                2.0 ** -900, 1.7e308], 400)
    p[:200] = 0.25  # equal neighbours: zero differences
    with np.errstate(all="ignore"):
        g, q = gradients(scn, p)
        assert np.array_equal(g, O.oracle_gradients(q, scn.shape, scn.mesh.dx), equal_nan=True)
