"""The direct sum and the energy on the integer pipes where their tiles, rows
and grid can go wrong: sizes around 128 and 256, uneven masses, and bodies off
the grid (no softening, a span of more than 2^13 softening lengths), which keep
the FP64 kernels. Against the oracle; 1e-12 as in test_diagnostics_gpu.py, for
accelerations relative to the largest one (terms round relative to themselves)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 127, 128, 129, 255, 257, 2049])
@pytest.mark.parametrize("eps,far", [(0.01, 0.0), (2.0, 0.0), (1e-5, 0.0), (0.0, 0.0), (0.01, 900.0)])
def test_sizes_and_both_paths(lib, orc, n, eps, far):
    b = lib.generate_ics(0, n, 17 + n)
    r = np.random.default_rng(n)
    b["mass"] *= 2.0 ** r.uniform(-30, 10, n)
    b["mass"][::11] = 0.0
    b["mass"][1] = 1.0
    b["x"][n - 1] += far
    idx = np.arange(n)
    sim = lib.Sim.from_bodies(b, softening=eps)
    got, (ke, pe) = sim.direct_forces(idx), sim.energy()
    sim.close()
    want = orc.direct_forces(b, 1.0, eps, idx)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    e = orc.total_energy(b, 1.0, eps)
    assert abs(ke + pe - e) <= 1e-12 * (abs(ke) + abs(pe))
