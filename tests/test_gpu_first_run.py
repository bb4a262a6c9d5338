"""The first run of a handle whose shape the autotuner knows (GB300 only): the fields of the following
runs bit for bit, and no wait for the making of the graph that those use."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import Solver, Sweep  # noqa: E402


def _sweep(n, nz, count, seed):
    return Sweep([W.plain_instance(n, nz, 5.0 + i + seed, 2.84, 50.0) for i in range(count)], crystal=W.CRYSTAL_QPM50)


@pytest.mark.parametrize("n,nz,count", [(16, 60, 1), (64, 30, 1), (128, 40, 2), (256, 60, 1), (256, 3, 1), (256, 40, 3)])
def test_first_run_has_the_bits_of_the_next(n, nz, count):
    for seed in range(3):  # the first handle of all runs the autotuner
        sw = _sweep(n, nz, count, seed)
        runs = []
        for _ in range(3):
            eta = sw.run()
            runs.append((eta, *sw.fields()))
        for eta, p, s in runs[1:]:
            assert np.allclose(eta, runs[0][0], rtol=1e-12, atol=0)
            assert all(np.array_equal(a, b) for a, b in zip(p + s, runs[0][1] + runs[0][2]))
        sw.close()


def test_first_run_after_a_change_of_inputs():
    """Given fields, then the Gaussian pump again: each change makes another graph."""
    n, nz = 256, 40
    inst = W.plain_instance(n, nz, 20.0, 2.84, 50.0)
    g = torch.Generator().manual_seed(1)
    pump = torch.randn(n, n, dtype=torch.complex64, generator=g).cuda()
    s = Solver(crystal=W.CRYSTAL_QPM50, nx=n, ny=n, nz=nz, lx=inst.lx, ly=inst.ly)
    out = []
    for _ in range(4):
        s.run(20.0, inst.waist, inst.focal, 50.0)
        a = s.fields()
        b = [v.cpu().numpy() for v in s.cwes_device(50.0, pump)]
        s.cwes_device(50.0, pump)
        out.append((*a, *b, s.efficiency()))
    for o in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(o[:4], out[0][:4]))
        assert abs(o[4] / out[0][4] - 1) < 1e-12
    s.close()


@pytest.mark.parametrize("n,nz,count", [(256, 400, 1), (128, 200, 2)])
def test_first_run_does_not_wait_for_a_graph(n, nz, count):
    """Median of seven new handles against their repeated runs. One launch instead of the streaming passes takes
    1.3 times their time, a new handle's own copies and allocations some hundredths: 1.5 is allowed."""
    first, later = [], []
    for seed in range(8):
        sw = _sweep(n, nz, count, seed)
        t = []
        for _ in range(4):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            sw.run()
            t.append(time.perf_counter() - t0)
        first.append(t[0])
        later.append(min(t[1:]))
        sw.close()
    assert np.median(first[1:]) < 1.5 * np.median(later[1:]), (first, later)
