"""Powers and efficiency belong to the handle's last run (GB300 only): a blocking run leaves them on
the host, an enqueued one (cwes_device) on the device, in any order of the two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import Solver  # noqa: E402


@pytest.mark.parametrize("n", [32, 64, 128])  # cluster march, cluster march, persistent grid
def test_powers_follow_the_last_run(n):
    inst = W.plain_instance(n, 12, 20.0, 2.84, 50.0)

    def solver():
        return Solver(crystal=W.CRYSTAL_QPM50, nx=n, ny=n, nz=12, lx=inst.lx, ly=inst.ly)

    g = torch.Generator().manual_seed(n)
    pump = torch.randn(n, n, dtype=torch.complex64, generator=g).cuda()
    other = solver()
    other.cwes_device(50.0, pump)
    torch.cuda.synchronize()
    eta_dev, pow_dev = other.efficiency(), other.powers()
    s = solver()
    etas = []
    for _ in range(2):
        s.run(20.0, inst.waist, 1000.0, 50.0)
        etas.append(s.efficiency())
        s.cwes_device(50.0, pump)
        torch.cuda.synchronize()
        # sums are FP64 atomics: order-dependent in the last bits
        np.testing.assert_allclose(s.efficiency(), eta_dev, rtol=1e-12)
        np.testing.assert_allclose(s.powers(), pow_dev, rtol=1e-12)
    np.testing.assert_allclose(etas[1], etas[0], rtol=1e-12)
    assert abs(etas[0] / eta_dev - 1) > 1e-3
