"""The blocked heat sweep on values its corrected products do not cover (GB300 only): a crystal at 0 C with
the beam's heat spreading into it, signed zeros, denormals, infinities and NaN, with the surroundings at
0 C and at 25 C, against the oracle's sweeps bit for bit (a NaN is a NaN), and what such a field costs."""
import ctypes as C
import time

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import _lib  # noqa: E402
from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import _cfg_from  # noqa: E402


def _sweeps(cfg, T, QK, t_inf, ns, bc):
    a, b, q = (torch.from_numpy(v).cuda() for v in (T, T, QK))
    torch.cuda.synchronize()
    t = time.perf_counter()
    _lib.check(_lib.lib().shg_heat_sweeps_device(C.byref(cfg), a.data_ptr(), b.data_ptr(), q.data_ptr(), t_inf, ns, bc,
                                                 torch.cuda.current_stream().cuda_stream), "shg_heat_sweeps_device")
    return (b if ns % 2 else a).cpu().numpy(), time.perf_counter() - t


def _same(a, b):
    nan = np.isnan(b)
    return np.array_equal(np.isnan(a), nan) and np.array_equal(a.view(np.uint32)[~nan], b.view(np.uint32)[~nan])


def _fields(kind, n, nz):
    x = np.linspace(-1, 1, n)
    beam = np.broadcast_to(np.exp(-40 * (x[:, None] ** 2 + x[None, :] ** 2)), (nz, n, n))
    T, Q = np.zeros((nz, n, n)), np.zeros((nz, n, n))
    if kind == "heated":  # values from the beam's to denormals and zeros
        Q = 5e-9 * beam
    elif kind == "cooled":  # the same below zero: fronts that underflow to -0
        Q = -5e-9 * beam
        T[nz // 3, n // 3, 2] = -1e-38
    elif kind == "signed":  # zeros of both signs, one value in two thousand
        T = np.where(np.arange(T.size).reshape(T.shape) % 3 == 0, -0.0, 0.0)
        T.flat[::2003] = 40.0
        Q = np.where(np.arange(T.size).reshape(T.shape) % 2 == 0, -0.0, 0.0)
    elif kind == "denormal":
        T = np.float32(1e-40) * (1 + np.arange(T.size).reshape(T.shape) % 7)
    elif kind == "small":  # products of the edges below 2^-102
        T = 10.0 ** -(30 + 8 * np.random.default_rng(2).random(T.shape))
    else:  # "nonfinite": ordinary temperatures with an infinity of either sign and a NaN
        T = 50 + beam
        T = np.array(T)
        T[nz // 2, n // 2, 3], T[nz // 2, 3, n // 2], T[1, n - 2, n - 2] = np.inf, -np.inf, np.nan
        Q = 5e-9 * beam
        Q = np.array(Q)
        Q[nz // 2 - 1, n // 4, n // 4] = np.nan
        Q[nz // 2 - 1, n // 4, 3 * n // 4] = np.inf
    return np.ascontiguousarray(T, np.float32), np.ascontiguousarray(Q, np.float32)


@pytest.mark.parametrize("kind", ["heated", "cooled", "signed", "denormal", "small", "nonfinite"])
@pytest.mark.parametrize("n,nz", [(40, 12), (64, 21), (136, 6)])
@pytest.mark.parametrize("bc", [0, 1])
def test_values_of_any_kind_bitexact(kind, n, nz, bc):
    T, Q = _fields(kind, n, nz)
    o = O.Oracle(O.make_cfg(W.CRYSTAL_QPM50, n, n, nz, 600.0, 500.0))
    cfg = _cfg_from(W.CRYSTAL_QPM50, nx=n, ny=n, nz=nz, lx=600.0, ly=500.0)
    with np.errstate(all="ignore"):
        QK = Q / np.float32(W.CRYSTAL_QPM50.kth)
        for t_inf in (0.0, 25.0):
            for ns in (1, 6):
                got, _ = _sweeps(cfg, T, QK, t_inf, ns, bc)
                assert _same(got, o.heat_sweeps(T, Q, t_inf, ns, bc)), (t_inf, ns)


@pytest.mark.parametrize("bc", [0, 1])
def test_a_crystal_at_zero_costs_little_more(bc):
    """128x128x200: a heated crystal that starts at 0 C against one at 50 C. Per voxel the range tests and the
    divisions of the smallest values are less than twice the work of a sweep in range; with the calls
    and the latency of the blocks that make them three times the time is allowed."""
    n, nz = 128, 200
    cfg = _cfg_from(W.CRYSTAL_QPM50, nx=n, ny=n, nz=nz, lx=600.0, ly=500.0)
    T, Q = _fields("heated", n, nz)
    zero = min(_sweeps(cfg, T, Q, 25.0, 200, bc)[1] for _ in range(5))
    warm = min(_sweeps(cfg, T + np.float32(50), Q, 25.0, 200, bc)[1] for _ in range(5))
    assert zero < 3 * warm, (zero, warm)
