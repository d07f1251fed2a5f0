"""Device memory of a handle: at most 2,010 bytes a body at 2,000,000 bodies. The
moments' sums live in the pool export's buffers, which a build does not need
otherwise, and the FP64 walk holds no copy of the cells."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
def test_bytes_per_body(lib, prec):
    torch = pytest.importorskip("torch")
    lib.Sim.from_bodies(lib.generate_ics(0, 1000, 1)).close()  # what a process holds once
    n = 2_000_000
    b = lib.generate_ics(2, n, 1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    sim = lib.Sim.from_bodies(b, softening=0.01, precision=prec)
    sim.substeps_async(1)
    sim.sync()
    held = before - torch.cuda.mem_get_info()[0]
    sim.close()
    assert held <= 2010 * n, held / n
