"""The FP32-mixed walk on both sides of the sizes up to which a system is summed by child
subtrees (5 tasks of 32 bodies per SM for opening angles of 0.45 or more, 8 below) and a
launch is split by them (7 tasks per SM in all).

Against the FP64 walk, errors relative to the largest acceleration, 1e-5; a system in
an ensemble has the bits it has alone, whichever launch either takes.
"""
import numpy as np
import pytest
import torch

from conftest import fields
from cosmosim_gb300.abi import BODY_DTYPE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm", [5, 7, 8])
@pytest.mark.parametrize("theta", [0.44, 0.45])
@pytest.mark.parametrize("over", [0, 1])
def test_both_sides(lib, per_sm, theta, over):
    n = 32 * per_sm * torch.cuda.get_device_properties(0).multi_processor_count + over
    b = lib.generate_ics(0, n, 50 + per_sm)
    got = []
    for prec in (1, 0):
        s = lib.Sim.from_bodies(b, softening=0.01, theta=theta, precision=prec)
        got.append(fields(s.bodies()))
        s.close()
    scale = np.linalg.norm(got[1], axis=1).max()
    assert np.linalg.norm(got[0] - got[1], axis=1).max() <= 1e-5 * scale
    other = lib.generate_ics(0, 17000, 3)  # past the launch's limit together
    for part in (other[:500], other):
        out = np.concatenate([b, part]).astype(BODY_DTYPE)
        ens = lib.Sim.ensemble(out, [n, len(part)], softening=0.01, theta=theta, precision=1)
        np.testing.assert_array_equal(fields(ens.bodies())[:n], got[0])
        ens.close()
