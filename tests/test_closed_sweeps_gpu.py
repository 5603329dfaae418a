"""The closed-form sweeps (the default kernels): every axis at line lengths
around the chunk, tile and launch-shape edges, in every precision mode, against
the oracle.  The bars are the suite's own: 1e-12 relative max-norm in FP64,
1e-6 for an FP32 field with FP64 arithmetic (a few roundings to FP32), 1e-5 in
FP32."""
import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from biofvm_b200._abi import FP32, FP32_FP64MATH, FP64
from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = {FP64: 1e-12, FP32_FP64MATH: 1e-6, FP32: 1e-5}


def run(scn, precision, steps=2):
    with Solver(0) as sv:
        load_scenario(sv, scn)
        if precision != FP64:
            sv.set_precision(precision)
            sv.set_densities(scn.initial_field())
        sv.set_grid_steps(False)
        sv.step(scn.dt, steps)
        return sv.get_densities()


# one point, partial and whole 16-point chunks, the change to 32-point chunks
# (a multiple of 32, or more than 160), the last length of 32-column tiles
# (256), two tensor boxes (257), the last 16-point shapes, the longest line
LENGTHS = [1, 2, 15, 16, 17, 32, 33, 64, 100, 160, 161, 192, 256, 257, 500, 512, 513, 1001, 1024]


@pytest.mark.parametrize("precision", [FP64, FP32_FP64MATH, FP32], ids=["fp64", "mixed", "fp32"])
@pytest.mark.parametrize("S", [1, 3, 4])
@pytest.mark.parametrize("n", LENGTHS)
def test_line_lengths(n, S, precision):
    for shape in ((n, 6, 5), (4, n, 5), (5, 4, n)):
        scn = W.mixed_small(shape=shape, S=S, n_agents=50, seed=n + S)
        got = run(scn, precision)
        err = O.max_rel_err(got, O.oracle_run(scn, 2, 7))
        assert np.all(err <= TOL[precision]), (shape, err)


@pytest.mark.parametrize("S", [2, 5, 7, 10, 11, 15, 16, 17, 33])
def test_density_counts(S):
    """Rows as tiles (several rows of S densities to a block's columns) and
    as plain columns; rows that are and are not 16-byte multiples."""
    for shape in ((64, 9, 4), (63, 9, 4), (256, 3, 2), (321, 5, 1)):
        scn = W.mixed_small(shape=shape, S=S, n_agents=60, seed=S)
        for precision in (FP64, FP32):
            err = O.max_rel_err(run(scn, precision), O.oracle_run(scn, 2, 7))
            assert np.all(err <= TOL[precision]), (shape, precision, err)


@pytest.mark.parametrize("D,dx", [(0.0, 10.0), (1e-3, 10.0), (1e5, 1.0), (1e7, 1.0)])
def test_slopes_from_zero_to_near_one(D, dx):
    """No diffusion (r = 0), hardly any, and c1 = dt D / dx^2 of 1e3 and 1e5.
    The elimination itself loses about c1 ulps of the field's mean in each
    solve (1 + 2 c1 + c2 is rounded), so the bar grows with c1: 6 solves of
    c1 2^-53 each, next to the 1e-12 of the moderate cases."""
    scn = W.mixed_small(shape=(40, 33, 70), S=2, n_agents=0, seed=5, dx=dx)
    scn.D = np.array([D, 0.5 * D])
    c1 = scn.dt * D / dx ** 2
    err = O.max_rel_err(run(scn, FP64), O.oracle_run(scn, 2, 7))
    assert np.all(err <= 1e-12 + 6 * c1 * 2.0 ** -53), err


def test_a_bad_value_stays_in_its_lines():
    """An infinity reaches the lines through its voxel and no other column."""
    scn = W.mixed_small(shape=(40, 20, 36), S=2, n_agents=0, seed=6, dirichlet=False, bulk=False)
    scn.p0[17 + 40 * (9 + 20 * 11), 0] = np.inf
    got = run(scn, FP64, steps=1)
    assert np.all(np.isfinite(got[:, 1]))
    clean = scn.p0.copy()
    clean[:, 0] = clean[:, 1]
    scn.p0 = clean
    assert np.array_equal(run(scn, FP64, steps=1)[:, 1], got[:, 1])


@pytest.mark.parametrize("shape,S", [((64, 64, 2), 1), ((50, 50, 50), 4), ((24, 24, 24), 20),
                                     ((64, 1, 64), 3), ((9, 64, 7), 9), ((17, 5, 64), 6),
                                     ((4, 4, 4), 300)])
def test_grid_steps_split_planes_by_densities(shape, S):
    """Planes of one item and of several, a last item with fewer densities,
    more items than SMs, and constants too many to stage: several steps in
    one launch against the oracle, agents sharing voxels included."""
    scn = W.mixed_small(shape=shape, S=S, n_agents=300, seed=sum(shape) + S)
    with Solver(0) as sv:
        load_scenario(sv, scn)
        assert sv.get_grid_steps() > 0
        sv.step(scn.dt, 3)
        err = O.max_rel_err(sv.get_densities(), O.oracle_run(scn, 3, 7))
    assert np.all(err <= TOL[FP64]), err


def test_many_row_tiles_a_place():
    """x rows enough for several blocks a place on the device (32,768 tiles)
    against the same step in slabs of 16 planes (2,048 tiles each, one block a
    place): the same tiles, the same bits."""
    rng = np.random.default_rng(11)
    shape, S = (96, 256, 256), 16
    scn = W.mixed_small(shape=shape, S=S, n_agents=0, seed=12, bulk=False, dirichlet=False)
    p = rng.uniform(0.5, 1.5, (int(np.prod(shape)), S))
    got = []
    for planes in (0, 16):
        with Solver(0) as sv:
            load_scenario(sv, scn)
            sv.set_densities(p)
            sv.set_slab_planes(planes)
            sv.step(scn.dt, 1)
            got.append(sv.get_densities())
    assert np.array_equal(got[0], got[1])
