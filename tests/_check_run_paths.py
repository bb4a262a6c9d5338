"""Child process of tests/test_gpu_check_paths.py (not collected): the SHG_CHECK build of the library (SHG_LIB) on the
kernels that its other child does not reach. The blocked heat sweep in tilings of large grids, in and out of
range; the single-sweep kernels by name and on an odd grid; persistent groups against the streaming
passes; the cluster march of 32 x 32 grids. Results are compared bit for bit, and no check may fail.
Prints one JSON line; exit status 0 when every comparison held."""
from __future__ import annotations

import ctypes as C
import json
import os
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path[:0] = [ROOT, HERE, os.path.join(ROOT, "oracle")]

import numpy as np  # noqa: E402
import torch  # noqa: E402

import oracle as O  # noqa: E402
from _util import bits_equal  # noqa: E402
from shg_focused_gaussian_beams_gb300 import _lib  # noqa: E402
from shg_focused_gaussian_beams_gb300 import solver as S  # noqa: E402
from shg_focused_gaussian_beams_gb300 import workloads as W  # noqa: E402

CR = W.CRYSTAL_QPM50
report = {"lib": _lib.LIB_PATH, "cases": {}}
ok = True


def record(name, good, **info):
    global ok
    ok &= bool(good)
    report["cases"][name] = {"ok": bool(good), **info}


def heat_fields(n, nz):
    rng = np.random.default_rng(n)
    T = (50 + rng.normal(0, 0.05, (nz, n, n))).astype(np.float32)
    return T, (rng.random(T.shape) * 5e-9).astype(np.float32)


def heat_cases():
    n, nz = 68, 21
    T, Q = heat_fields(n, nz)
    QK = Q / np.float32(CR.kth)
    o = O.Oracle(O.make_cfg(CR, n, n, nz, 600.0, 500.0))
    cfg = S._cfg_from(CR, nx=n, ny=n, nz=nz, lx=600.0, ly=500.0)
    zero = T.copy()
    zero[9, 20, 20] = 0.0
    for bc in (0, 1):
        for levels in (1, 2):
            for threads, vx, zc in ((256, 8, 7), (512, 32, 17), (256, 16, 1)):
                for name, f in (("", T), (":zero", zero)):
                    a, b, q = (torch.from_numpy(v).cuda() for v in (f, f, QK))
                    _lib.check(_lib.lib().shg_check_heat_tiling(C.byref(cfg), a.data_ptr(), b.data_ptr(), q.data_ptr(), 25.0, 1, bc,
                                                                levels, threads, vx, zc, None), "tiling")
                    record(f"tiling{levels}/{threads}/{vx}/{zc}:bc{bc}{name}",
                           bits_equal(b.cpu().numpy(), o.heat_sweeps(f, Q, 25.0, levels, bc)))
    for kind, n in (("tma", 40), ("ws4", 40), ("", 33)):
        os.environ.pop("SHG_HEAT", None)
        if kind:
            os.environ["SHG_HEAT"] = kind
        T, Q = heat_fields(n, 12)
        for bc in (0, 1):
            want = O.Oracle(O.make_cfg(CR, n, n, 12, 600.0, 500.0)).heat_sweeps(T, Q, 25.0, 3, bc)
            record(f"heat{n}{kind}:bc{bc}", bits_equal(S.heat_sweeps(CR, T, Q, 25.0, 3, bc, lx=600.0, ly=500.0), want))
    os.environ.pop("SHG_HEAT", None)


def schedule_cases():
    for n, nzs in ((64, [9, 4, 2, 12]), (128, [5, 7]), (256, [4, 3])):
        insts = [W.plain_instance(n, nz, 5.0 + i, 2.84, 50.0) for i, nz in enumerate(nzs)]
        f = {}
        for kind in ("group", False):
            sw = S.Sweep(insts, crystal=CR)
            sw.set_schedule(n, resident=kind)
            f[kind] = sw.run(with_fields=True)[1]
            sw.close()
        record(f"group{n}", all(bits_equal(a, b) for a, b in zip(f["group"], f[False])))
    for n, count in ((32, 1), (32, 40), (64, 1), (64, 20), (128, 10)):
        insts = [W.plain_instance(n, 8, 5.0 + i, 2.84, 50.0) for i in range(count)]
        f = {}
        for kind in ("cluster", "streaming"):
            os.environ["SHG_MARCH"] = f"{n}:{kind}"
            sw = S.Sweep(insts, crystal=CR)
            f[kind] = sw.run(with_fields=True)[1]
            label = sw.schedule()
            sw.close()
            record(f"schedule{n}x{count}:{kind}", kind[:7] in label, label=label)
        record(f"cluster{n}x{count}", all(bits_equal(a, b) for a, b in zip(f["cluster"], f["streaming"])))
    os.environ.pop("SHG_MARCH", None)


heat_cases()
schedule_cases()
e, s, v = C.c_int(), C.c_int(), C.c_longlong()
_lib.check(_lib.lib().shg_check_status(C.byref(e), C.byref(s), C.byref(v)), "shg_check_status")
record("no_failed_check", e.value == 1 and s.value == 0, site=s.value, value=v.value)
print(json.dumps(report))
sys.exit(0 if ok else 1)
