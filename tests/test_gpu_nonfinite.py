"""A nonlinear coefficient that is not a number is not a crystal without coupling (GB300 only): the
fields come out as NaN and the efficiency is refused, on every schedule."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300._lib import ShgError  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import Solver  # noqa: E402


@pytest.mark.parametrize("march", ["64:streaming", "64:coop", "64:cluster", "64:1/1"])
@pytest.mark.parametrize("deff", [float("nan"), float("inf")])
def test_nonfinite_coupling_is_reported(deff, march, monkeypatch):
    monkeypatch.setenv("SHG_MARCH", march)
    inst = W.plain_instance(64, 8, 20.0, 2.84, 50.0)
    s = Solver(crystal=dataclasses.replace(W.CRYSTAL_QPM50, deff=deff), nx=64, ny=64, nz=8, lx=inst.lx, ly=inst.ly)
    s.run(inst.power, inst.waist, inst.focal, inst.temp)
    p, sh = s.fields()
    assert np.all(np.isnan(p.real)) and np.all(np.isnan(sh.real))
    with pytest.raises(ShgError):
        s.efficiency()
    s.close()
