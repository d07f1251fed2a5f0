"""Cell moments where the fixed-point sums would lose bits: those systems, and only
those, take the FP64 sums.

A system has the bits it has alone, whatever its neighbours in the handle are (a body of
1e-20 of the system's mass, a light body close to the origin, extreme extents). Centres of
mass of light cells close to the origin: within (n + 3) 2^-53 of the sum of the
magnitudes (n products and sums and a division in FP64), against extended precision.
"""
import numpy as np
import pytest

from conftest import fields
from cosmosim_gb300.abi import BODY_DTYPE

pytestmark = pytest.mark.gpu

LD = np.longdouble


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


@pytest.mark.parametrize("mass", [2.0 ** -20, 2.0 ** -49])
@pytest.mark.parametrize("scale", [2.0 ** -27, 2.0 ** -40, 2.0 ** -52])
def test_light_cells_close_to_the_origin(lib, mass, scale):
    r = np.random.default_rng(8)
    b = np.zeros(64, dtype=BODY_DTYPE)
    for f in "xyz":
        b[f] = r.uniform(-1.0, 1.0, 64)
        b[f][:32] = scale * r.uniform(0.5, 1.0, 32)
    b["mass"] = 1.0
    b["mass"][:32] = mass * r.uniform(0.5, 1.0, 32)
    pool, size = lib.octree_build(b)
    x = np.stack([b[f] for f in "xyz"], 1)
    checked = 0
    for c in pool[:size]:
        if c["half_size"] > 4 * scale:
            continue  # may hold others
        centre = np.array([c["center_x"], c["center_y"], c["center_z"]])
        inside = np.flatnonzero((np.abs(x[:32] - centre) <= c["half_size"]).all(1))
        k = len(inside)
        if k < 2 or not np.isclose(c["total_mass"], b["mass"][inside].sum(), rtol=1e-12):
            continue
        m = b["mass"][inside].astype(LD)
        for d, f in enumerate(("cx", "cy", "cz")):
            want = (m * x[inside, d].astype(LD)).sum() / m.sum()
            assert abs(LD(c[f]) - want) <= (k + 3) * 2.0 ** -53 * want, (f, k)
        checked += 1
    assert checked >= 8
