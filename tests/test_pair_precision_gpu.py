"""Accuracy of one body's acceleration, and of the energy, where a sum or a difference
held in too few bits would show: close pairs near the origin of a wide system, a heavy
body among light ones, systems of very different masses in one handle, masses just
below a power of two.

Against extended precision over all pairs (theta 0). Errors are relative to the sum of
the terms' magnitudes. Bar: n pairs in FP64, each term within 4 roundings (difference,
m/r^3, product), the sums in any order within one a term: (n + 8) 2^-53.
"""
import numpy as np
import pytest

from conftest import fields
from cosmosim_gb300.abi import BODY_DTYPE

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
LD = np.longdouble


def bodies(x, m):
    b = np.zeros(len(m), dtype=BODY_DTYPE)
    for d, f in enumerate("xyz"):
        b[f] = x[:, d]
    b["mass"] = m
    return b


def near_pair(sep, far, seed):
    """Two bodies about sep apart and from the origin, a third one far out."""
    r = np.random.default_rng(seed)
    x = r.normal(size=(3, 3))
    x /= np.linalg.norm(x, axis=1)[:, None]
    x *= np.array([0.5 * sep, 0.5 * sep, far])[:, None] * r.uniform(0.7, 1.0, (3, 1))
    return bodies(x, r.uniform(0.5, 1.0, 3))


def heavy_among_light(seed):
    r = np.random.default_rng(seed)
    x = r.normal(size=(1001, 3))
    return bodies(x, np.where(np.arange(1001) == 500, 1.0, 1e-12 * r.uniform(0.5, 1.0, 1001)))


def exact(b, eps):
    """Accelerations, the terms' magnitudes and the pair energies in extended precision."""
    x = np.stack([b[f] for f in "xyz"], 1).astype(LD)
    m = b["mass"].astype(LD)
    acc, mag = np.zeros((len(b), 3), LD), np.zeros(len(b), LD)
    e2 = LD(eps * eps)
    pe = LD(0)
    for i in range(len(b)):
        d = x - x[i]
        r2 = (d * d).sum(1) + e2
        w = m / (r2 * np.sqrt(r2))
        w[i] = 0
        t = d * w[:, None]
        acc[i], mag[i] = t.sum(0), np.sqrt((t * t).sum(1)).sum()
        pe -= (m[i] * m[i + 1:] / np.sqrt(r2[i + 1:])).sum()
    return acc, mag, pe


def errors(got, acc, mag):
    d = got.astype(LD) - acc
    return np.sqrt((d * d).sum(1)) / mag


def scenes():
    for eps, far in ((0.01, 5.0), (0.01, 40.0), (0.01, 80.0), (0.3, 80.0), (0.01, 2e4), (1e-6, 5.0)):
        for sep in (1e-2, 1e-3, 1e-4, 1e-6):
            yield eps, [near_pair(sep, far, s) for s in range(20)]
    for eps in (1e-2, 1e-3):
        yield eps, [heavy_among_light(s) for s in range(3)]


def test_walk(lib):
    for eps, systems in scenes():
        for b in systems:
            s = lib.Sim.from_bodies(b, softening=eps, theta=0.0, precision=0)
            err = errors(fields(s.bodies()), *exact(b, eps)[:2])
            s.close()
            assert err.max() <= (len(b) + 8) * U, (eps, float(err.max()))


def test_direct_sum(lib):
    for eps, systems in scenes():
        for b in systems:
            s = lib.Sim.from_bodies(b, softening=eps)
            err = errors(s.direct_forces(np.arange(len(b))), *exact(b, eps)[:2])
            s.close()
            assert err.max() <= (len(b) + 8) * U, (eps, float(err.max()))


def test_direct_sum_and_energy_of_systems_of_unequal_mass(lib):
    parts = [near_pair(0.1, 4.0, 1), near_pair(0.1, 4.0, 2), near_pair(0.1, 4.0, 3)]
    for p, w in zip(parts, (1.0, 1e-25, 1e12)):
        p["mass"] *= w
    s = lib.Sim.ensemble(np.concatenate(parts).astype(BODY_DTYPE), [3, 3, 3], softening=0.01)
    got, (_, pe) = s.direct_forces(np.arange(9)), s.energy()
    s.close()
    want = LD(0)
    for g, p in enumerate(parts):
        acc, mag, e = exact(p, 0.01)
        assert errors(got[3 * g:3 * g + 3], acc, mag).max() <= 11 * U, g
        want += e
    assert abs(LD(pe) - want) <= 19 * U * abs(want)


def test_energy(lib):
    for eps, systems in scenes():
        for b in systems:
            s = lib.Sim.from_bodies(b, softening=eps)
            pe = s.energy()[1]
            s.close()
            want = exact(b, eps)[2]
            assert abs(LD(pe) - want) <= (len(b) + 8) * U * abs(want), (eps, pe)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -7, 2.0 ** 5])
def test_energy_of_full_mantissas(lib, scale):
    """Masses just below a power of two, distances just below one: the largest
    significand a pair term can have."""
    eps = 1.0 - 3e-7
    r = np.random.default_rng(9)
    parts = []
    for _ in range(256):
        x = np.zeros((2, 3))
        x[1, 0] = 8e-4 * np.sqrt(r.random())
        parts.append(bodies(x * scale, scale * np.array([1.0 - U, 1.0 - U])))
    s = lib.Sim.ensemble(np.concatenate(parts).astype(BODY_DTYPE), [2] * 256, softening=eps * scale)
    pe = s.energy()[1]
    s.close()
    want = sum(exact(p, eps * scale)[2] for p in parts)
    assert abs(LD(pe) - want) <= 264 * U * abs(want)
