"""Row passes of the batched THERMAL pass (GB300 only): the block shape follows the batch size and
the reverse sweep enters a segment in the pass that leaves the one above it. Neither changes an
operation or its order, so the results are the same bits for every batch size and checkpoint
count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402
from shg_focused_gaussian_beams_gb300.solver import ThermalGradBatch  # noqa: E402


def batch(n, nz, count):
    inst = W.plain_instance(n, nz, 20.0, 2.84, 50.0)
    T = np.broadcast_to(50 + 0.3 * np.linspace(0, 1, nz)[:, None, None], (nz, n, n)).astype(np.float32).copy()
    T += 0.1 * np.cos(np.arange(n, dtype=np.float32))[None, None, :]
    tb = ThermalGradBatch(count, crystal=W.CRYSTAL_QPM50, nx=n, ny=n, nz=nz, lx=inst.lx, ly=inst.ly)
    for i in range(count):
        tb.set_temperature(i, T, 20.0 + (i % 2), inst.waist, 1000.0)
    return tb


# one solve, one past the first limit of the rule (152 blocks of the narrow shape) and past the second
@pytest.mark.parametrize("n,counts", [(16, (153, 310)), (32, (77, 155)), (64, (20, 39)), (128, (10, 20)), (256, (3, 5))])
def test_batch_size_does_not_change_a_solve(n, counts):
    nz = 4
    one = batch(n, nz, 1)
    pump = one.gaussian_pumps()
    f1 = one.forward(pump, with_fields=True)
    f1 = {k: v.clone() for k, v in f1.items() if torch.is_tensor(v)}
    g1 = one.gradient(pump, checkpoints=2)["grad"].clone()
    for count in counts:
        tb = batch(n, nz, count)
        p = tb.gaussian_pumps()
        f = tb.forward(p, with_fields=True)
        g = tb.gradient(p, checkpoints=2)["grad"]
        for i in (0, (count - 1) // 2 * 2):  # solves with the first one's power
            assert torch.equal(f["pump_out"][i], f1["pump_out"][0]) and torch.equal(f["sh_out"][i], f1["sh_out"][0])
            assert torch.equal(g[i], g1[0])


@pytest.mark.parametrize("nz", [2, 3, 11])
def test_segments_do_not_change_the_gradient(nz):
    tb = batch(32, nz, 2)
    p = tb.gaussian_pumps()
    want = tb.gradient(p, checkpoints=nz)["grad"].clone()
    for checkpoints in range(1, nz):
        assert torch.equal(tb.gradient(p, checkpoints=checkpoints)["grad"], want), checkpoints
