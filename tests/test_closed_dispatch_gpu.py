"""Which kernel sweeps an axis, and that a change of it keeps the results:
the closed form by default, the tabulated kernels where a path, a
configuration, fused sources or a length past 1024 points asks for them, and
the chunk length following added densities after a first step.  Steps against
the oracle at the suite's 1e-12."""
import dataclasses

import numpy as np
import pytest

from biofvm_b200 import Solver, load_scenario
from biofvm_b200 import workloads as W
from biofvm_b200._abi import PATH_AUTO, PATH_TMA
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def swept(sv):
    return [sv.get_closed_sweep(ax) for ax in range(3)]


def closed(sv):
    return [c > 0 for c in swept(sv)]


def check_step(sv, scn):
    step = dataclasses.replace(scn, p0=sv.get_densities())
    sv.step(scn.dt, 1)
    err = O.max_rel_err(sv.get_densities(), O.oracle_run(step, 1, 7))
    assert np.all(err <= 1e-12), err


@pytest.mark.parametrize("shape,S", [((96, 20, 12), 4), ((160, 12, 10), 5), ((64, 20, 12), 6)])
def test_what_sweeps_an_axis(shape, S):
    scn = W.mixed_small(shape=shape, S=S, n_agents=200, seed=sum(shape) + S)
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.set_grid_steps(False)
        assert closed(sv) == [True] * 3
        check_step(sv, scn)
        for path, expect in ((PATH_TMA, [False] * 3), (PATH_AUTO, [True] * 3)):
            sv.set_kernel_path(path)
            assert closed(sv) == expect
            check_step(sv, scn)
        sv.set_fuse_sources(True)
        assert closed(sv) == [False, True, True]
        check_step(sv, scn)
        sv.set_fuse_sources(False)
        sv.set_sweep_config(1, 8, 16)
        assert closed(sv) == [True, False, True]
        check_step(sv, scn)


def test_long_lines_and_coefficients():
    scn = W.mixed_small(shape=(1100, 5, 4), S=2, n_agents=50, seed=4)
    with Solver(0) as sv:
        load_scenario(sv, scn)
        assert closed(sv) == [False, True, True]
        check_step(sv, scn)
        sv.set_coefficients(np.array([1.0, -1.0]), np.zeros(2))
        sv.reset_diffusion_setup()
        sv.step(scn.dt, 1)
        assert closed(sv) == [False] * 3


def test_chunks_follow_an_added_density():
    """x of 64 points takes 16-point chunks while 32-point ones would leave
    fewer than 128 threads an SM (15,360 in all with one density, 30,720 with
    two), 32-point chunks from the second density on."""
    scn = W.mixed_small(shape=(64, 96, 80), S=2, n_agents=0, seed=8, bulk=False, dirichlet=False)
    m = scn.mesh
    with Solver(0) as sv:
        sv.resize_densities(1)
        sv.resize_space(m.x0, m.x1, m.y0, m.y1, m.z0, m.z1, m.dx, m.dy, m.dz)
        sv.set_coefficients(scn.D[:1], scn.decay[:1])
        sv.set_densities(scn.p0[:, :1])
        sv.set_grid_steps(False)
        first = sv.get_closed_sweep(0)
        sv.step(scn.dt, 1)
        sv.add_density(float(scn.D[1]), float(scn.decay[1]))
        assert (first, sv.get_closed_sweep(0)) == (16, 32)
        p = sv.get_densities()
        p[:, 1] = scn.p0[:, 1]
        sv.set_densities(p)
        check_step(sv, scn)


def test_an_axis_goes_back_to_the_default():
    """After a set configuration and after the tuner, with the fields of a
    solver that never left the default."""
    scn = W.mixed_small(shape=(40, 36, 130), S=2, n_agents=100, seed=21)
    with Solver(0) as sv, Solver(0) as plain:
        for s in (sv, plain):
            load_scenario(s, scn)
            s.set_grid_steps(False)
        shapes = [sv.get_sweep_config(ax) for ax in range(3)]
        for ax in range(3):
            sv.set_sweep_config(ax, 16, 16, 2)
        assert swept(sv) == [0, 0, 0]
        for ax in range(3):
            sv.reset_sweep_config(ax)
        assert swept(sv) == swept(plain) == [16, 16, 16]
        assert [sv.get_sweep_config(ax) for ax in range(3)] == shapes
        sv.step(scn.dt, 2)
        sv.tune_sweeps(scn.dt, 1)
        sv.set_fuse_sources(False)
        for ax in range(3):
            sv.reset_sweep_config(ax)
        sv.set_slab_planes(0)
        assert swept(sv) == [16, 16, 16]
        sv.step(scn.dt, 1)
        plain.step(scn.dt, 3)
        got = sv.get_densities()
        assert np.array_equal(got, plain.get_densities())
    err = O.max_rel_err(got, O.oracle_run(scn, 3, 7))
    assert np.all(err <= 1e-12), err


def test_the_tuner_times_the_default_x_sweep_with_fusion_set():
    """x of this field takes 31 us in closed form and 49 us in the best of the
    tabulated kernels: the tuner must find it also where sources were set to be
    fused into x (there is nothing to fuse, so that setting stays)."""
    scn = W.mixed_small(shape=(161, 97, 123), S=3, n_agents=0, seed=9, bulk=False)
    with Solver(0) as sv:
        load_scenario(sv, scn)
        sv.set_fuse_sources(True)
        sv.tune_sweeps(scn.dt, 10)
        assert sv.get_fuse_sources() and sv.get_closed_sweep(0) == 0
        sv.set_fuse_sources(False)
        assert sv.get_closed_sweep(0) > 0
