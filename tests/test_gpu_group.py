"""Persistent groups of blocks (the "group" schedule) against the streaming passes: the same
arithmetic, so the output fields are equal bit for bit (GB300 only). Fewer solves than groups, as
many and more (the queue), uneven lengths down to the shortest march, several classes at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import Sweep  # noqa: E402


def _fields(insts, grids, kind):
    sw = Sweep(insts, crystal=W.CRYSTAL_QPM50)
    for n in grids:
        sw.set_schedule(n, resident=kind)
    eta = sw.run()
    eta2 = sw.run()
    assert np.allclose(eta, eta2, rtol=1e-13, atol=0)
    p, s = sw.fields()
    sw.close()
    return eta, p, s


@pytest.mark.parametrize("n,nzs", [(64, [2, 3, 17, 30]), (64, [9] * 230), (128, [2, 21, 8]), (128, [5] * 90),
                                   (256, [2]), (256, [7, 3] * 13)])
def test_groups_match_streaming(n, nzs):
    insts = [W.plain_instance(n, nz, 3.0 + i % 7, 1.0 + 0.1 * (i % 9), 50.0) for i, nz in enumerate(nzs)]
    eg, pg, sg = _fields(insts, [n], "group")
    es, ps, ss = _fields(insts, [n], False)
    assert np.allclose(eg, es, rtol=1e-12, atol=0)
    for a, b in zip(pg + sg, ps + ss):
        assert np.array_equal(a, b)


def test_groups_of_three_classes_run_together():
    insts = [W.plain_instance([64, 128, 256][i % 3], 4 + i, 10.0, 2.0, 50.0) for i in range(12)]
    _, pg, sg = _fields(insts, [64, 128, 256], "group")
    _, ps, ss = _fields(insts, [64, 128, 256], False)
    for a, b in zip(pg + sg, ps + ss):
        assert np.array_equal(a, b)


def test_groups_are_refused_on_other_grids():
    from shg_focused_gaussian_beams_gb300._lib import ShgError
    sw = Sweep([W.plain_instance(32, 5, 5.0, 2.0, 50.0)] * 2, crystal=W.CRYSTAL_QPM50)
    with pytest.raises(ShgError):
        sw.set_schedule(32, resident="group")
