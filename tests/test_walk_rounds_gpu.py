"""The walks' rounds (32 cells of a warp's stack at a time) where they can go
wrong: tasks of few bodies, remainders of 32, one-cell trees, opening angles
from "nothing is accepted" on, and trees whose open cells outgrow the stack.

Against the oracle's walk on the oracle's tree. A body's error is taken
relative to the largest acceleration: a term rounds relative to itself (FP64
about 2^-52, FP32-mixed about 2^-22), so a body whose terms cancel is as exact
as the others only in that sense. FP64 1e-11, FP32-mixed 1e-5. Interaction
totals are equal.
"""
import numpy as np
import pytest

from conftest import fields
from cosmosim_gb300.abi import BODY_DTYPE

pytestmark = pytest.mark.gpu


def lattice(k, seed):
    """k^3 bodies, one per cell of a full octree (k a power of two): every
    opened cell has eight children."""
    r = np.random.default_rng(seed)
    g = (np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) / k
    p = g + r.uniform(-0.2, 0.2, g.shape) / k
    b = np.zeros(len(p), dtype=BODY_DTYPE)
    for d, f in enumerate("xyz"):
        b[f] = p[:, d]
    b["mass"] = r.uniform(0.5, 2.0, len(p))
    return b


def check(lib, orc, b, theta, eps=0.01):
    from cosmosim_gb300.lib import Sim

    pool, _ = orc.octree_build(b)
    want = b.copy()
    orc.octree_compute_forces(pool, want, 1.0, eps, theta)
    count, _ = orc.count_interactions(pool, b, theta)
    scale = max(np.linalg.norm(fields(want), axis=1).max(), 1e-300)
    for prec, tol in ((0, 1e-11), (1, 1e-5)):
        s = Sim.from_bodies(b, softening=eps, theta=theta, precision=prec)
        err = np.linalg.norm(fields(s.bodies()) - fields(want), axis=1).max() / scale
        s.enable_stats(True)
        s.build_tree_async()
        s.gravity_async()
        hits = s.interactions()
        got = fields(s.bodies())
        s.close()
        assert err <= tol, (prec, err)
        assert np.linalg.norm(got - fields(want), axis=1).max() <= tol * scale, prec
        assert hits == count, prec


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 97, 4097])
@pytest.mark.parametrize("theta", [0.0, 0.3, 0.7, 1.2])
def test_small_and_ragged_systems(lib, orc, n, theta):
    check(lib, orc, lib.generate_ics(0, n, 40 + n), theta)


@pytest.mark.parametrize("n", [33, 2049, 70001])
@pytest.mark.parametrize("eps", [1e-5, 40.0])
def test_softenings_off_and_far_inside_the_grid(lib, orc, n, eps):
    """The FP64 walk's pair terms run on integers while the span is at most
    2^13 softening lengths, else in FP64 (the first of the two)."""
    check(lib, orc, lib.generate_ics(0, n, 60), 0.5, eps)


@pytest.mark.parametrize("k", [16, 32])
def test_full_octree_with_every_cell_opened(lib, orc, k):
    check(lib, orc, lattice(k, 7), 0.0)


@pytest.mark.parametrize("eps", [0.01, 1e-5])
def test_ensemble_systems_equal_themselves_alone(lib, eps):
    """FP64: 72,000 bodies in systems of 9,000 take several child subtrees of the
    root per unit, one system alone one: the same bits, on the grid and off."""
    from cosmosim_gb300.lib import Sim

    parts = [lib.generate_ics(3, 9000, 80 + g) for g in range(8)]
    out = np.zeros(72000, dtype=BODY_DTYPE)
    for g, p in enumerate(parts):
        out[9000 * g:9000 * (g + 1)] = p
    ens = Sim.ensemble(out, [9000] * 8, softening=eps)
    got = fields(ens.bodies())
    ens.close()
    for g in (0, 5):
        one = Sim.from_bodies(parts[g], softening=eps)
        np.testing.assert_array_equal(got[9000 * g:9000 * (g + 1)], fields(one.bodies()))
        one.close()


@pytest.mark.parametrize("theta", [0.0, 0.5])
@pytest.mark.parametrize("spoil", ["no", "far", "heavy"])
def test_caller_pool_walks(lib, orc, theta, spoil):
    """octree_compute_forces on a pool that the oracle built (its child table is
    made by the import), also with a cell far outside the bodies' box or heavier
    than its children."""
    b = lattice(8, 3)
    pool, _ = orc.octree_build(b)
    if spoil == "far":
        pool["cx"][70] = 1e4
    elif spoil == "heavy":
        pool["total_mass"][9] = 1e9
    want = b.copy()
    orc.octree_compute_forces(pool, want, 1.0, 0.02, theta)
    lib.octree_compute_forces(pool, b, 1.0, 0.02, theta)
    scale = np.linalg.norm(fields(want), axis=1).max()
    assert np.linalg.norm(fields(b) - fields(want), axis=1).max() <= 1e-11 * scale
