"""The FP64 walk on both sides of the sizes up to which it is split by child subtrees
(6 tasks of 32 bodies per SM for opening angles of 0.45 or more, 12 below).

Against the oracle's walk on the oracle's tree, errors relative to the largest
acceleration, 1e-11; a system in an ensemble has the bits it has alone.
"""
import numpy as np
import pytest
import torch

from conftest import fields
from cosmosim_gb300.abi import BODY_DTYPE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm", [6, 12])
@pytest.mark.parametrize("theta", [0.44, 0.45])
@pytest.mark.parametrize("over", [0, 1])
def test_both_sides(lib, orc, per_sm, theta, over):
    from cosmosim_gb300.lib import Sim

    n = 32 * per_sm * torch.cuda.get_device_properties(0).multi_processor_count + over
    b = lib.generate_ics(0, n, 30 + per_sm)
    pool, _ = orc.octree_build(b)
    want = b.copy()
    orc.octree_compute_forces(pool, want, 1.0, 0.01, theta)
    scale = np.linalg.norm(fields(want), axis=1).max()
    s = Sim.from_bodies(b, softening=0.01, theta=theta, precision=0)
    got = fields(s.bodies())
    s.close()
    assert np.linalg.norm(got - fields(want), axis=1).max() <= 1e-11 * scale
    small = lib.generate_ics(0, 500, 3)
    out = np.concatenate([b, small]).astype(BODY_DTYPE)
    ens = Sim.ensemble(out, [n, 500], softening=0.01, theta=theta, precision=0)
    np.testing.assert_array_equal(fields(ens.bodies())[:n], got)
    ens.close()
