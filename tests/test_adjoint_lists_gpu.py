"""The adjoint's lists where their layout changes: few bodies, remainders of 32,
and both sides of the size (about 38,800 bodies on 152 SMs) up to which a task's
list walk is shared out by segments; cells of up to 8, up to 256 and more bodies.

The run is the FP64 handle's up to rounding (1e-11 of the largest coordinate);
the gradient's derivative along one direction agrees with the central
difference of the frozen map (step 1e-6: truncation and rounding below 1e-5).
"""
import numpy as np
import pytest

from conftest import fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 300, 2049, 38000, 39500])
def test_run_and_gradient(lib, n):
    b = lib.generate_ics(0, n, 11 + n)
    kw = dict(softening=0.02, theta=0.5)
    adj = lib.Adjoint(n, dt=1e-3, substeps=2, checkpoint_every=2, **kw)
    x0 = fields(b, ("x", "y", "z"))
    r = np.random.default_rng(n)
    target = x0 + r.normal(0.0, 0.1, x0.shape)
    _, got = adj.forward(b, target, record=True, final=True)
    gx, _ = adj.backward()
    s = lib.Sim.from_bodies(b, dt=1e-3, precision=0, **kw)
    s.substeps_async(2)
    want = fields(s.bodies(), ("x", "y", "z"))
    s.close()
    assert np.abs(fields(got, ("x", "y", "z")) - want).max() <= 1e-11 * np.abs(x0).max()
    d = r.normal(size=x0.shape)
    h, loss = 1e-6, []
    for sign in (1.0, -1.0):
        c = b.copy()
        for q, f in enumerate("xyz"):
            c[f] += sign * h * d[:, q]
        loss.append(adj.forward_frozen(c, target))
    adj.close()
    fd = (loss[0] - loss[1]) / (2 * h)
    assert abs(fd - (gx * d).sum()) <= 1e-5 * max(abs(fd), np.abs(gx * d).sum())
