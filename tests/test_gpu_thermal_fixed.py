"""Stage phases of the batched THERMAL pass at large rotation angles (GB300 only): with few
slices and a detuned poling period a quarter step of the phase mismatch is above and below
half a radian (the series and the sincosf branch of its rotation), up to a few radians.

Tolerance: the FP32 oracle's own phases round to ulp(|phase|), at most 4e-6 rad here, and the
fields to a few 1e-7 per step over at most 8 steps: 2e-5 relative is an order above their sum."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from _util import rel_l2

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import ThermalGradBatch  # noqa: E402


@pytest.mark.parametrize("nz", [2, 3, 9])
@pytest.mark.parametrize("detune", [1.0, 1.0005, 1.003, 0.99])
def test_rotation_angles(nz, detune):
    n = 32
    cr = dataclasses.replace(W.CRYSTAL_QPM50, lambda_qpm=float(np.float32(W.CRYSTAL_QPM50.lambda_qpm * detune)), lz=2000.0)
    inst = W.plain_instance(n, nz, 20.0, 2.84, 50.0)
    o = O.Oracle(O.make_cfg(cr, n, n, nz, inst.lx, inst.ly))
    z = np.linspace(0, 1, nz)[:, None, None]
    T = np.broadcast_to(50 + 0.3 * z, (nz, n, n)).astype(np.float32).copy()
    tb = ThermalGradBatch(1, crystal=cr, nx=n, ny=n, nz=nz, lx=inst.lx, ly=inst.ly)
    tb.set_temperature(0, T, 20.0, inst.waist, 1000.0)
    pump = tb.gaussian_pumps()
    f = tb.forward(pump, with_fields=True)
    p = pump[0].cpu().numpy()
    po, so = o.cwes_thermal(T, p, np.zeros_like(p), float(T[0, n // 2, n // 2]))
    assert rel_l2(f["pump_out"][0].cpu().numpy(), po) < 2e-5
    assert rel_l2(f["sh_out"][0].cpu().numpy(), so) < 2e-5
