"""The blocked heat sweep in tilings that the planner takes on large grids only (GB300 only): one and two sweeps
per launch, 256 and 512 threads, whole rows and tiles in x and y, chunks that fill the plane ring more than
once, ragged last chunks, and values out of range that appear planes into a chunk; small grids against the
oracle, the planner's own choices on large ones against the single-sweep kernel, bit for bit."""
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


def _cfg(n, nz):
    return _cfg_from(W.CRYSTAL_QPM50, nx=n, ny=n, nz=nz, lx=600.0, ly=500.0)


def _fields(n, nz, seed):
    rng = np.random.default_rng(seed)
    T = (50 + rng.normal(0, 0.05, (nz, n, n))).astype(np.float32)
    Q = (rng.random(T.shape) * 5e-9).astype(np.float32)
    return T, Q


def _tiled(n, nz, T, QK, launches, bc, levels, threads, vx, zc):
    a, b, q = (torch.from_numpy(v).cuda() for v in (T, T, QK))
    cfg = _cfg(n, nz)
    _lib.check(_lib.lib().shg_check_heat_tiling(C.byref(cfg), a.data_ptr(), b.data_ptr(), q.data_ptr(), 25.0, launches, bc, levels,
                                                threads, vx, zc, torch.cuda.current_stream().cuda_stream), "tiling")
    return (b if launches % 2 else a).cpu().numpy()


# n, nz, vectors a row, planes a chunk: whole rows (vx >= n / 4) and tiles in x, whole columns and tiles in y
TILINGS = [(64, 41, 16, 5), (64, 41, 16, 8), (64, 41, 32, 17), (72, 23, 32, 7), (100, 30, 16, 17), (68, 19, 8, 7), (128, 18, 32, 18)]


@pytest.mark.parametrize("n,nz,vx,zc", TILINGS)
@pytest.mark.parametrize("threads", [256, 512])
@pytest.mark.parametrize("levels", [1, 2])
@pytest.mark.parametrize("bc", [0, 1])
def test_tilings_bitexact(n, nz, vx, zc, threads, levels, bc):
    T, Q = _fields(n, nz, n + zc)
    # out of range a few planes into a chunk: a zero, a denormal beside it, a huge value in another tile
    far = T.copy()
    far[(zc + 3) % nz, n // 2, n // 3] = 0.0
    far[(zc + 3) % nz, n // 2 + 1, n // 3] = 1e-40
    far[nz - 2, n // 5, n - 3] = 1e35
    o = O.Oracle(O.make_cfg(W.CRYSTAL_QPM50, n, n, nz, 600.0, 500.0))
    QK = Q / np.float32(W.CRYSTAL_QPM50.kth)
    for field in (T, far):
        for launches in (1, 2):
            got = _tiled(n, nz, field, QK, launches, bc, levels, threads, vx, zc)
            assert bits_equal(got, o.heat_sweeps(field, Q, 25.0, launches * levels, bc)), (launches, field is far)


@pytest.mark.parametrize("n,nz", [(128, 200), (160, 120), (200, 150), (228, 90), (256, 400)])
@pytest.mark.parametrize("bc", [0, 1])
def test_the_planners_choice_on_large_grids(n, nz, bc, monkeypatch):
    T, Q = _fields(n, nz, nz)
    for f in ("ordinary", "zeros"):
        if f == "zeros":
            T = T * (np.arange(nz) % 40 > 20).astype(np.float32)[:, None, None]
        out = {}
        for kind in (None, "ws4"):
            monkeypatch.delenv("SHG_HEAT", raising=False)
            if kind:
                monkeypatch.setenv("SHG_HEAT", kind)
            a, b, q = (torch.from_numpy(v).cuda() for v in (T, T, Q))
            cfg = _cfg(n, nz)
            _lib.check(_lib.lib().shg_heat_sweeps_device(C.byref(cfg), a.data_ptr(), b.data_ptr(), q.data_ptr(), 25.0, 7, bc,
                                                         torch.cuda.current_stream().cuda_stream), "sweeps")
            out[kind] = (b.cpu().numpy(), a.cpu().numpy())  # the result of seven, and the state before the last
        assert bits_equal(out[None][0], out["ws4"][0]) and bits_equal(out[None][1], out["ws4"][1]), f


def test_no_tiling_is_refused():
    T, Q = _fields(64, 8, 1)
    a, b, q = (torch.from_numpy(v).cuda() for v in (T, T, Q))
    st = torch.cuda.current_stream().cuda_stream
    cfg = _cfg(64, 8)
    call = lambda *t, shift=0: _lib.lib().shg_check_heat_tiling(C.byref(cfg), a.data_ptr() + shift, b.data_ptr(), q.data_ptr(),  # noqa: E731
                                                                25.0, 0, 0, *t, st)
    assert call(1, 256, 16, 4) == 0
    for t in [(0, 256, 16, 4), (3, 256, 16, 4), (1, 128, 16, 4), (1, 256, 12, 4), (1, 256, 64, 4), (1, 256, 4, 4),
              (1, 256, 16, 0), (1, 256, 16, 9)]:
        assert call(*t) == 1, t
    assert call(1, 256, 16, 4, shift=4) == 1
