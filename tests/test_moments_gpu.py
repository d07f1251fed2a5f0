"""Cell masses and centres of mass from prefix sums, where they can go wrong: tiles
of 256 bodies and their remainders, masses too unequal for the fixed-point sums
(which then are not used), systems far from the origin, coincident bodies.

Against the oracle's pool (FP64 sums): centres within 1e-12 of the distance from
the origin, masses within 1e-13. Two builds give the same bits.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(lib, orc, b):
    got, size = lib.octree_build(b)
    want, wsize = orc.octree_build(b)
    assert size == wsize
    got, want = got[:size], want[:size]
    np.testing.assert_array_equal(got["body_index"], want["body_index"])
    np.testing.assert_allclose(got["total_mass"], want["total_mass"], rtol=1e-13, atol=0)
    big = np.abs(np.stack([b[f] for f in "xyz"])[:, b["mass"] > 0]).max() if size else 1.0
    for f in ("cx", "cy", "cz"):
        assert np.abs(got[f] - want[f]).max() <= 1e-12 * big, f
    again, _ = lib.octree_build(b)
    for f in ("cx", "cy", "cz", "total_mass"):
        np.testing.assert_array_equal(again[f][:size], got[f])


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 511, 513, 4096, 70001])
def test_sizes(lib, orc, n):
    b = lib.generate_ics(0, n, 21)
    b["mass"] *= np.random.default_rng(n).uniform(0.5, 2.0, n)
    check(lib, orc, b)


@pytest.mark.parametrize("low", [1e-3, 1e-11, 1e-17, 1e-40, 1e-310])
@pytest.mark.parametrize("scale", [1.0, 1e-120, 1e60])
def test_unequal_masses(lib, orc, low, scale):
    r = np.random.default_rng(5)
    b = lib.generate_ics(0, 3000, 22)
    b["mass"] = scale * np.exp(r.uniform(np.log(max(low, 1e-300)), 0.0, 3000))
    b["mass"][7] = low * scale
    check(lib, orc, b)


def test_far_from_the_origin_and_coincident(lib, orc):
    b = lib.generate_ics(0, 3000, 23)
    for f in "xyz":
        b[f][100:160] = b[f][100]
        b[f][400:500] *= 1e-9
        b[f] += 1e4
    check(lib, orc, b)
