"""Cluster march by cluster size (GB300 only): the size follows the number of solves of the class, and
does not change a result: fields as the streaming passes, bit for bit, on repeated runs (each from
zeroed SH fields)."""
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
    for _ in range(2):
        eta, f = sw.run(with_fields=True)
    f = [np.array(x) for x in f]
    sw.close()
    return eta, f


# both sizes of each grid, at one solve, in one wave, and at more solves than a wave holds
@pytest.mark.parametrize("n,count", [(64, 1), (64, 18), (64, 19), (64, 37), (64, 60), (128, 8), (128, 9), (128, 17),
                                     (128, 30), (256, 2), (256, 12)])
def test_cluster_sizes_match_streaming(n, count):
    insts = [W.plain_instance(n, 3 + i % 4, 3.0 + i % 7, 1.0 + 0.1 * (i % 9), 50.0) for i in range(count)]
    ec, fc = _fields(insts, n, "cluster")
    es, fs = _fields(insts, n, False)
    np.testing.assert_allclose(ec, es, rtol=1e-12, atol=0)
    for a, b in zip(fc, fs):
        assert np.array_equal(a, b)


# sizes that the schedule call does not name: the variable fixes the kind, the count the cluster size
@pytest.mark.parametrize("n,count", [(32, 1), (32, 36), (32, 40), (32, 74), (32, 80), (32, 160), (64, 8), (64, 9)])
def test_small_grids_match_streaming(monkeypatch, n, count):
    insts = [W.plain_instance(n, 2 + i % 4, 3.0 + i % 7, 1.0 + 0.1 * (i % 9), 50.0) for i in range(count)]
    es, fs = _fields(insts, n, False)
    monkeypatch.setenv("SHG_MARCH", f"{n}:cluster")
    sw = Sweep(insts, crystal=W.CRYSTAL_QPM50)
    assert "cluster march" in sw.schedule()
    for _ in range(2):
        ec, fc = sw.run(with_fields=True)
    np.testing.assert_allclose(ec, es, rtol=1e-12, atol=0)
    for a, b in zip(fc, fs):
        assert np.array_equal(a, b)
    sw.close()
