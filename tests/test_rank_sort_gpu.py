"""The counting sort of small builds, against the oracle's tree (which inserts
bodies in index order): sizes around its tiles, its groups of 32 and its upper
limit, coincident bodies (equal keys keep index order) and massless ones.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 128, 129, 1023, 1024, 1025, 2049, 12287,
                               12288, 12289])
def test_build_equals_the_oracles(lib, orc, n):
    r = np.random.default_rng(n)
    b = lib.generate_ics(0, n, 3)
    k = r.permutation(n)[:n // 5]
    for f in ("x", "y", "z"):
        b[f][k] = b[f][k[::-1]] if len(k) else b[f][k]  # pairs at one place
    b["mass"][r.permutation(n)[:n // 16]] = 0.0
    got, size = lib.octree_build(b)
    want, wsize = orc.octree_build(b)
    assert size == wsize
    for f in got.dtype.names:
        if got[f].dtype.kind == "i":
            np.testing.assert_array_equal(got[f][:size], want[f][:size], err_msg=f)
