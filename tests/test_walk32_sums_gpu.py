"""The FP32-mixed walk's sums: uncompensated chains of at most 8 additions.

One body feels 512 to 4,096 others at one place (to FP32), every cell opened, so all terms
are the same number f, which a run with one of them gives. Up to 8 equal terms, or up to
16 two by two, are within 2.5 x 2^-24 of their exact sum in FP32 (the largest over
all significands and counts; 16 one by one: 4.5); the compensation keeps what the sum
of the blocks rounds away.
"""
import numpy as np
import pytest

from cosmosim_gb300.abi import BODY_DTYPE

pytestmark = pytest.mark.gpu


def system(k, mass, seed):
    r = np.random.default_rng(seed)
    b = np.zeros(k + 1, dtype=BODY_DTYPE)
    b["mass"] = mass
    b["mass"][0] = 1.0
    b["x"][1:] = 1.0 + 1e-9 * r.uniform(-1, 1, k)
    b["y"][1:], b["z"][1:] = 1e-9 * r.uniform(-1, 1, (2, k))
    return b


@pytest.mark.parametrize("k", [512, 4096])
def test_equal_terms(lib, k):
    r = np.random.default_rng(k)
    worst = 0.0
    for t in range(200):
        mass = r.uniform(1.0, 2.0)
        a = []
        for n in (1, k):
            s = lib.Sim.from_bodies(system(n, mass, t), softening=0.01, theta=0.0, precision=1)
            a.append(s.bodies()["ax"][0])
            s.close()
        worst = max(worst, abs(a[1] / (k * a[0]) - 1.0))
    assert worst <= 2.6 * 2.0 ** -24, worst * 2.0 ** 24
