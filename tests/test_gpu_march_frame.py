"""The plain march's scaled frame at the edges of its rule (GB300 only): no coupling at all, a
very small coupling, and a negative one, from given pump and SH fields, on the
streaming, persistent and cluster-resident schedules, against the oracle.

Tolerance: FIELD_RTOL, the parity bar of every other march test; without coupling the two fields
only diffract and are absorbed, so an SH that started at zero must stay exactly zero."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from _util import FIELD_RTOL, rel_l2, smooth_noise

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import Solver  # noqa: E402


@pytest.mark.parametrize("march", ["64:streaming", "64:coop", "64:cluster", "64:1/1"])
@pytest.mark.parametrize("deff", [0.0, 1e-13, -6.75e-6, 6.75e-6])
def test_coupling_edges(deff, march, monkeypatch):
    monkeypatch.setenv("SHG_MARCH", march)
    n, nz = 64, 12
    cr = dataclasses.replace(W.CRYSTAL_QPM50, deff=deff, lambda_qpm=float(np.float32(W.CRYSTAL_QPM50.lambda_qpm * 1.001)))
    inst = W.plain_instance(n, nz, 20.0, 2.84, 50.0)
    o = O.Oracle(O.make_cfg(cr, n, n, nz, inst.lx, inst.ly))
    rng = np.random.default_rng(5)
    p = (o.set_pump(inst.power, inst.focal, inst.waist, inst.temp) * (1 + 0.1 * smooth_noise(rng, n))).astype(np.complex64)
    for s in ((0.3 * p * np.exp(0.4j)).astype(np.complex64), np.zeros_like(p)):
        sol = Solver(crystal=cr, nx=n, ny=n, nz=nz, lx=inst.lx, ly=inst.ly)
        sol.set_input_fields(p, s)
        sol.cwes(inst.temp)
        po, so = sol.fields()
        pr, sr, _, _ = o.cwes_plain(p, s, inst.temp)
        assert rel_l2(po, pr) < FIELD_RTOL
        if np.any(sr):
            assert rel_l2(so, sr) < FIELD_RTOL
        else:
            assert not np.any(so)
