"""Systems with a few bodies far out: the walks then share out the subtrees below
a deeper cell than the root, and the FP64 walk's integer pair terms take far
cells from a coarser grid (up to a span of 2^21 softening lengths), tasks with a
far body in FP64.

Against the oracle's walk on the oracle's tree, errors relative to the largest
acceleration: FP64 1e-11, FP32-mixed 1e-5, interaction totals equal.
"""
import numpy as np
import pytest

from conftest import fields
from cosmosim_gb300.abi import BODY_DTYPE

pytestmark = pytest.mark.gpu

EPS = 0.01


def scattered(lib, n, span, seed=5, share=0.04):
    """A disk, every 25th body (at least one) thrown out to span softenings."""
    b = lib.generate_ics(0, n, seed)
    r = np.random.default_rng(seed)
    k = r.permutation(n)[:max(1, int(share * n))]
    d = r.normal(size=(len(k), 3))
    d *= span * EPS * r.uniform(0.01, 1.0, len(k))[:, None] / np.abs(d).max(1)[:, None]
    d[0] *= span * EPS / np.abs(d[0]).max()
    for q, f in enumerate("xyz"):
        b[f][k] = d[:, q]
    return b


@pytest.mark.parametrize("n", [2, 33, 2049, 20000, 70001])
@pytest.mark.parametrize("span", [2.0 ** 13.5, 2.0 ** 17, 2.0 ** 20.9, 2.0 ** 24])
def test_against_the_oracle(lib, orc, n, span):
    from cosmosim_gb300.lib import Sim

    b = scattered(lib, n, span)
    pool, _ = orc.octree_build(b)
    want = b.copy()
    orc.octree_compute_forces(pool, want, 1.0, EPS, 0.5)
    count, _ = orc.count_interactions(pool, b, 0.5)
    scale = np.linalg.norm(fields(want), axis=1).max()
    for prec, tol in ((0, 1e-11), (1, 1e-5)):
        s = Sim.from_bodies(b, softening=EPS, theta=0.5, precision=prec)
        err = np.linalg.norm(fields(s.bodies()) - fields(want), axis=1).max() / scale
        s.enable_stats(True)
        s.build_tree_async()
        s.gravity_async()
        hits = s.interactions()
        s.close()
        assert err <= tol, (prec, err)
        assert hits == count, prec


@pytest.mark.parametrize("prec", [0, 1])
def test_ensemble_systems_equal_themselves_alone(lib, prec):
    from cosmosim_gb300.lib import Sim

    spans = [2.0 ** 10, 2.0 ** 14, 2.0 ** 19, 2.0 ** 24, 2.0 ** 16, 2.0 ** 18, 2.0 ** 22, 2.0 ** 12]
    parts = [scattered(lib, 9000, s, 80 + g) for g, s in enumerate(spans)]
    out = np.zeros(72000, dtype=BODY_DTYPE)
    for g, p in enumerate(parts):
        out[9000 * g:9000 * (g + 1)] = p
    ens = Sim.ensemble(out, [9000] * 8, softening=EPS, precision=prec)
    got = fields(ens.bodies())
    ens.close()
    for g in (0, 1, 2, 3, 6):
        one = Sim.from_bodies(parts[g], softening=EPS, precision=prec)
        np.testing.assert_array_equal(got[9000 * g:9000 * (g + 1)], fields(one.bodies()))
        one.close()
