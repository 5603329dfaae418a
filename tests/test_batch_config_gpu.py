"""A member's sweep configuration changed between two steps of a batch on
branches: the captured graph must follow the kernel that sweeps each axis and
the chunk length its Dirichlet segments are laid out for.  Against the oracle
at the suite's bar for one instance (1e-12 relative max-norm)."""
import dataclasses

import numpy as np
import pytest

from biofvm_b200 import Batch, Solver, load_scenario
from biofvm_b200 import workloads as W
from biofvm_b200._abi import BATCH_BRANCHES, PATH_GENERIC, PATH_TMA
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def reported_y(sv, dt):
    sv.set_sweep_config(1, *sv.get_sweep_config(1)[:3])


def slabs(sv, dt):
    sv.set_slab_planes(4)


def tuned(sv, dt):
    sv.tune_sweeps(dt, 1)


# y of 128 or 130 points: 16-point chunks in the closed form, 32-point chunks
# in the tabulated kernels (fewer segments, in the same buffers)
@pytest.mark.parametrize("shape,S,change", [((24, 130, 20), 2, reported_y),
                                            ((64, 128, 12), 1, reported_y),
                                            ((24, 130, 20), 2, slabs),
                                            ((40, 36, 9), 3, tuned)])
def test_a_member_changes_its_sweeps_between_two_steps(shape, S, change):
    scns = [W.mixed_small(shape=shape, S=S, n_agents=200, seed=sum(shape) + S),
            W.mixed_small(shape=(20, 30, 10), S=1, n_agents=50, seed=3)]
    sols = [Solver(0) for _ in scns]
    try:
        for sv, scn in zip(sols, scns):
            load_scenario(sv, scn)
        with Batch(0) as bt:
            for sv in sols:
                bt.add(sv)
            bt.set_mode(BATCH_BRANCHES)
            bt.step(scns[0].dt, 2)
            bt.synchronize()
            change(sols[0], scns[0].dt)
            bt.step(scns[0].dt, 2)
            bt.synchronize()
            got = [sv.get_densities() for sv in sols]
    finally:
        for sv in sols:
            sv.close()
    for scn, p in zip(scns, got):
        err = O.max_rel_err(p, O.oracle_run(scn, 4, 7))
        assert np.all(err <= 1e-12), (scn.shape, err)


@pytest.mark.parametrize("route", ["default", "configured", "tma", "register"])
def test_new_coefficients_between_two_steps(route):
    """The diffusion setup is reset and made anew from other coefficients: the
    graph's kernels must read the new tables, tabulated ones among them."""
    scns = [W.mixed_small(shape=(24, 40, 20), S=2, n_agents=100, seed=31),
            W.mixed_small(shape=(20, 30, 10), S=1, n_agents=50, seed=3)]
    sols = [Solver(0) for _ in scns]
    try:
        for sv, scn in zip(sols, scns):
            load_scenario(sv, scn)
        if route == "configured":
            sols[0].set_sweep_config(2, 8, 16)
        elif route != "default":
            sols[0].set_kernel_path(PATH_TMA if route == "tma" else PATH_GENERIC)
        with Batch(0) as bt:
            for sv in sols:
                bt.add(sv)
            bt.set_mode(BATCH_BRANCHES)
            for _ in range(2):  # the second replays what the first one's tables settled
                bt.step(scns[0].dt, 2)
            bt.synchronize()
            scn = dataclasses.replace(scns[0], D=scns[0].D[::-1] * 3.0, decay=scns[0].decay + 0.5,
                                      p0=sols[0].get_densities())
            sols[0].set_coefficients(scn.D, scn.decay)
            sols[0].reset_diffusion_setup()
            bt.step(scn.dt, 2)
            bt.synchronize()
            err = O.max_rel_err(sols[0].get_densities(), O.oracle_run(scn, 2, 7))
            other = O.max_rel_err(sols[1].get_densities(), O.oracle_run(scns[1], 6, 7))
    finally:
        for sv in sols:
            sv.close()
    assert np.all(err <= 1e-12) and np.all(other <= 1e-12), (err, other)
