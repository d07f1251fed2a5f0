"""The SPH pass of a handle's substep (neighbour lists from the sorted bodies)
where its tiles can go wrong: body counts around a chunk of 32 and a
super-chunk of 1024, coincident bodies (one depth-64 leaf names only its
first), few and only gas, spheres that hold everything or nothing. A step of
dt = 0 leaves the positions as they are, so density, pressure and smoothing
length must equal the oracle's bit for bit; accelerations (gravity on this
library's tree plus the SPH sums) to 1e-11 of the largest."""
import numpy as np
import pytest

from cosmosim_gb300.abi import NODE_DTYPE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 64, 1023, 1024, 1025, 3100])
@pytest.mark.parametrize("gas,h", [(1.0, 0.0), (0.05, 0.0), (1.0, 1e-6), (0.5, 60.0)])
def test_sph_of_a_still_step_equals_the_oracle(lib, orc, n, gas, h):
    b = lib.generate_ics(1, n, 900 + n)
    r = np.random.default_rng(n)
    is_gas = r.random(n) < gas
    is_gas[n - 1] = True
    b["type"] = np.where(is_gas, 1, 0)
    b["smoothing_h"] = h if h else r.uniform(0.05, 2.0, n)
    b["internal_energy"] = r.uniform(0.05, 1.0, n)
    b["mass"] = r.uniform(0.5, 2.0, n) / n
    if n > 40:  # coincident bodies, a dead one among them
        for f in "xyz":
            b[f][10:14] = b[f][3]
        b["mass"][12] = 0.0
    want = b.copy()
    pool = np.zeros(8 * n, dtype=NODE_DTYPE)
    orc.integrator_step(want, 0.0, 1.0, 0.01, 0.5, pool, 1)
    sim = lib.Sim.from_bodies(b, softening=0.01, dt=0.0, sph=True)
    sim.substeps_async(1)
    got = sim.bodies()
    sim.close()
    for f in ("density", "pressure", "smoothing_h", "internal_energy"):
        np.testing.assert_array_equal(got[f], want[f], err_msg=f)
    scale = max(np.abs(want[f]).max() for f in ("ax", "ay", "az"))
    for f in ("ax", "ay", "az"):
        assert np.abs(got[f] - want[f]).max() <= 1e-11 * scale, f
