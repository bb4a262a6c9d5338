"""The blocked heat sweep (one or two sweeps per launch, the default where NX % 4 == 0) against
the oracle's sweeps, bit for bit (GB300 only): grids at the edges of its tiles, sweep counts
around pairs, both boundary modes, and values outside the range of its corrected products."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from _util import bits_equal

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import _lib  # noqa: E402
from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import _cfg_from  # noqa: E402


def _device_sweeps(n, nz, T, QK, ns, bc):
    cfg = _cfg_from(W.CRYSTAL_QPM50, nx=n, ny=n, nz=nz, lx=600.0, ly=500.0)
    a, b, q = (torch.from_numpy(v).cuda() for v in (T, T, QK))
    _lib.check(_lib.lib().shg_heat_sweeps_device(C.byref(cfg), a.data_ptr(), b.data_ptr(), q.data_ptr(), 25.0, ns, bc,
                                                 torch.cuda.current_stream().cuda_stream), "shg_heat_sweeps_device")
    out = (b, a) if ns % 2 else (a, b)
    return out[0].cpu().numpy(), out[1].cpu().numpy()


# whole rows of 2, 4, 8, 16, 32 vectors; tiles in x with one or two ragged ends; NZ of one chunk, of
# ragged chunks, and the smallest
@pytest.mark.parametrize("n,nz", [(8, 2), (12, 3), (16, 24), (36, 7), (64, 21), (68, 5), (100, 9), (128, 6), (300, 5)])
@pytest.mark.parametrize("bc", [0, 1])
def test_blocked_sweeps_bitexact(n, nz, bc):
    """Both buffers: the result of `ns` sweeps and the state before the last one."""
    o = O.Oracle(O.make_cfg(W.CRYSTAL_QPM50, n, n, nz, 600.0, 500.0))
    rng = np.random.default_rng(n + nz)
    T = (o.init_temperature(48.0, 50.0, 46.5, bc) + rng.normal(0, 0.05, (nz, n, n))).astype(np.float32)
    Q = (rng.random(T.shape) * 5e-9).astype(np.float32)
    QK = Q / np.float32(W.CRYSTAL_QPM50.kth)
    for ns in (1, 2, 3, 6):
        got, before = _device_sweeps(n, nz, T, QK, ns, bc)
        assert bits_equal(got, o.heat_sweeps(T, Q, 25.0, ns, bc)), ns
        assert bits_equal(before, o.heat_sweeps(T, Q, 25.0, ns - 1, bc) if ns > 1 else T), ns


@pytest.mark.parametrize("scale", [0.0, 1e-25, 1e34, -1.0])
@pytest.mark.parametrize("bc", [0, 1])
def test_values_outside_the_corrected_range(scale, bc):
    """A field of zeros, of magnitudes below 2^-60 or above 2^99, and of negative temperatures, with
    one hot voxel of ordinary magnitude."""
    n, nz = 40, 12
    o = O.Oracle(O.make_cfg(W.CRYSTAL_QPM50, n, n, nz, 600.0, 500.0))
    rng = np.random.default_rng(3)
    T = ((50 + rng.random((nz, n, n))) * scale).astype(np.float32)
    T[nz // 2, n // 2, 7] = 51.0
    Q = np.zeros_like(T)
    got, _ = _device_sweeps(n, nz, T, Q, 5, bc)
    assert bits_equal(got, o.heat_sweeps(T, Q, 25.0, 5, bc))
