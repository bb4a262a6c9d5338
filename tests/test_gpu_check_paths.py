"""The SHG_CHECK build (device-side index checks) on the blocked heat sweep's long chunks, the single-sweep heat
kernels, the persistent groups and the cluster marches, in a child process (GB300 only); no check may
fail."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - CPU containers
    pytest.skip("no CUDA device", allow_module_level=True)

from shg_focused_gaussian_beams_gb300 import build as B  # noqa: E402

HERE = os.path.dirname(os.path.abspath(__file__))


def test_paths_under_index_checks():
    lib = B.build(variant="check")
    r = subprocess.run([sys.executable, os.path.join(HERE, "_check_run_paths.py")], env=dict(os.environ, SHG_LIB=lib),
                       capture_output=True, text=True, timeout=600)
    assert r.stdout.strip(), r.stderr[-3000:]
    report = json.loads(r.stdout.strip().splitlines()[-1])
    bad = {k: v for k, v in report["cases"].items() if not v["ok"]}
    assert r.returncode == 0 and not bad, (bad, r.stderr[-2000:])
    assert os.path.samefile(report["lib"], lib)
