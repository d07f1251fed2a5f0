"""Cell moments where the fixed-point sums would lose bits: those systems, and only
those, take the FP64 sums.

A system has the bits it has alone, whatever its neighbours in the handle are (a body of
1e-20 of the system's mass, a light body close to the origin, extreme extents).
"""
import numpy as np
import pytest

from conftest import fields
from cosmosim_gb300.abi import BODY_DTYPE

pytestmark = pytest.mark.gpu


def odd_system(lib, kind, n=3000):
    b = lib.generate_ics(0, n, 33)
    if kind == "light":
        b["mass"][11] = 1e-20 * b["mass"].sum()
    elif kind == "near":  # light, and 1e-13 of the extent from the origin
        b["mass"][11] = 1e-12 * b["mass"].sum()
        for f in "xyz":
            b[f][11] = 1e-13
    elif kind == "wide":
        for f in "xyz":
            b[f] *= 1e100
    return b


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("kind", ["light", "near", "wide"])
def test_neighbours_do_not_change_a_system(lib, prec, kind):
    if kind == "wide" and prec == 1:
        pytest.skip("beyond FP32 positions")
    plain = [lib.generate_ics(0, 5000, 40), lib.generate_ics(2, 4001, 41)]
    for p in plain:
        p["mass"] *= np.random.default_rng(6).uniform(0.5, 2.0, len(p))
    parts = [plain[0], odd_system(lib, kind), plain[1]]
    sim = lib.Sim.ensemble(np.concatenate(parts).astype(BODY_DTYPE), [len(p) for p in parts],
                           softening=0.01, precision=prec)
    got = np.split(fields(sim.bodies()), np.cumsum([len(p) for p in parts])[:-1])
    sim.close()
    for p, a in zip(parts, got):
        one = lib.Sim.from_bodies(p, softening=0.01, precision=prec)
        np.testing.assert_array_equal(a, fields(one.bodies()))
        one.close()
