"""Line transforms on split lanes (GB300 only): the lone-solve passes of 128- and 256-point lines
(persistent grid, one-solve streaming launches, THERMAL march) compute a DFT's even and odd outputs on two
lanes. Every output takes the butterflies of the unsplit transform with the same roundings, so the
fields equal those of the passes that do not split (the persistent groups) bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import Sweep  # noqa: E402


def _fields(insts, n, kind):
    sw = Sweep(insts, crystal=W.CRYSTAL_QPM50)
    sw.set_schedule(n, resident=kind)
    _, f = sw.run(with_fields=True)
    f = [np.array(x) for x in f]
    sw.close()
    return f


@pytest.mark.parametrize("n", [64, 128, 256])  # 64: the largest line that is not split
@pytest.mark.parametrize("nz", [2, 3, 20])
def test_lone_solve_matches_unsplit_passes(n, nz):
    insts = [W.plain_instance(n, nz, p, xi, 50.0) for p, xi in ((10.0, 2.84), (45.0, 0.6))]
    pair = _fields(insts, n, "group")
    for i, inst in enumerate(insts):
        for kind in ("coop", False):
            (one,) = _fields([inst], n, kind)
            assert np.array_equal(one, pair[i])
