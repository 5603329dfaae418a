"""The adjoint's dot products and agent updates against the tangent-linear
model at the edges of their segments: columns of 1, 4 k, 8 k and 8 k + 1
points, rows of one voxel, densities that do not divide a block, more items
than threads on the device, and one voxel shared by many agents.  Both sides
are exact derivatives of one discrete map in FP64: 1e-9 relative."""
import numpy as np
import pytest

from biofvm_b200 import workloads as W
from biofvm_b200.adjoint import AdjointProblem
from oracle import tangent_linear as TL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,S,agents,flags", [
    ((16, 8, 24), 1, 40, 7),
    ((5, 17, 9), 3, 300, 7),
    ((1, 4, 25), 7, 20, 7),
    ((33, 1, 1), 2, 200, 6),
    ((70, 65, 64), 9, 500, 7),
    ((3, 3, 3), 100, 60, 7),
])
def test_adjoint_at_segment_edges(shape, S, agents, flags):
    steps = 2
    scn = W.mixed_small(shape=shape, S=S, n_agents=agents, seed=sum(shape) + S)
    th = (np.array(scn.agent_secretion, float), np.array(scn.agent_uptake, float),
          np.array(scn.D, float), np.array(scn.decay, float))
    rng = np.random.default_rng(5)
    v = [x * rng.uniform(0.5, 1.5, x.shape) for x in th]
    target = rng.uniform(0, 2, (scn.num_voxels, S))
    prob = AdjointProblem(scn, steps, checkpoint_every=2, flags=flags)
    try:
        p = prob.forward(*th)
        g = prob.backward(p - target)
    finally:
        prob.close()
    # one parameter group at a time, so that no group hides in another's sum
    for i, key in enumerate(("secretion", "uptake", "D", "decay")):
        only = [x if j == i else np.zeros_like(x) for j, x in enumerate(v)]
        pt, pd = TL.tangent_run(scn, steps, flags, *th, *only)
        dL = np.sum((pt - target) * pd)
        scale = np.sum(np.abs((pt - target) * pd))
        assert abs(np.sum(g[key] * v[i]) - dL) <= 1e-9 * scale, key
