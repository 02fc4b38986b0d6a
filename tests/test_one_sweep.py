"""Float 16384-point transforms: one cluster sweep in calls of up to 2^25 points, two
passes above and wherever a thread count or split is cached, and in the split
tensor-core form.  Schedules and routes on the CPU emulator; calls on both sides of
the line, of one aux, on the GPU against FP64 (bar: 1e-6 log2 N).
"""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N = 16384

CHILD = r'''
import ctypes, json, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from notorious_fft import Library
L = Library(sys.argv[2])
cluster, lean = L.lib.nfft_emu_cluster_launches, L.lib.nfft_emu_lean_launches
cluster.restype = lean.restype = ctypes.c_longlong
x = np.random.default_rng(1).standard_normal((3, 16384, 2)).astype(np.float32).view(np.complex64)[..., 0]
y = np.zeros_like(x)
with L.mkaux("dft", [16384]) as a:
    before = cluster(), lean()
    a.batched("dft", x, y, 3, 16384, 16384)
    want = np.fft.fft(x.astype(complex))
    print(json.dumps(dict(split=a.schedule()[0], logt=a.schedule()[1], cluster=cluster() - before[0],
                          lean=lean() - before[1], err=float(np.linalg.norm(y - want) / np.linalg.norm(want)))))
'''


@pytest.mark.parametrize("entry,split,logt,one", [(None, [7, 7], 0, True), (([], 8), [7, 7], 8, False),
                                                  (([], 7), [7, 7], 7, False), (([8, 6], 0), [8, 6], 0, False),
                                                  (([14], 0), [7, 7], 0, True)])
def test_schedules(emu_f, tmp_path, entry, split, logt, one):
    cache = tmp_path / "tune.json"
    rows = [{"device": "emulated sm_100 sm_100 driver 0", "key": f"f32:plan:dft:{N}", "split": entry[0],
             "logt": entry[1], "us": 1.0}] if entry else []
    cache.write_text('{"format": "notorious_fft tune cache 1", "entries": [\n' +
                     ",\n".join(json.dumps(r) for r in rows) + "\n]}\n")
    r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "notorious-fft_b200"),
                        os.path.join(ROOT, "tests", "emu", "_build", "libnfft_emu_f.so")],
                       env=dict(os.environ, NOTORIOUS_FFT_TUNE_CACHE=str(cache)), capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    got = json.loads(r.stdout.strip().splitlines()[-1])
    assert (got["split"], got["logt"]) == (split, logt)
    assert (got["cluster"], got["lean"]) == ((1, 0) if one else (0, 2))
    assert got["err"] <= 1e-6 * 14


@pytest.mark.gpu
def test_both_sides_of_the_line(lib_f):
    import torch
    from notorious_fft import FORM_SPLIT_TC
    x = torch.randn(2049, N, dtype=torch.complex64, device="cuda")
    want = torch.fft.fft(x.to(torch.complex128))
    with lib_f.mkaux("dft", [N]) as aux:
        for batch, launches in ((2048, 1), (2049, 2), (1, 1), (2048, 1)):
            y = torch.zeros_like(x)
            before = lib_f.launch_count()
            aux.batched("dft", x, y, batch, N, N)
            torch.cuda.synchronize()
            assert lib_f.launch_count() - before == launches
            err = (y[:batch] - want[:batch]).norm() / want[:batch].norm()
            assert err <= 1e-6 * 14 and not y[batch:].any()
        aux.set_form(FORM_SPLIT_TC)
        y = torch.zeros_like(x)
        before = lib_f.launch_count()
        aux.batched("dft", x, y, 2049, N, N)
        torch.cuda.synchronize()
        assert lib_f.launch_count() - before == 2
        assert (y - want).norm() / want.norm() <= 2e-6
