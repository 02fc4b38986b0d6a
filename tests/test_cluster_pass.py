"""Passes whose tile is shared by a cluster of CTAs: 8192-point (double) and
16384-point (float) lines, and the 1024- and 2048-point strided axes, with line
counts that end inside a tile, padded distances, both directions and in place; on
the CPU emulator (bounds-checked) and on the GPU, against the oracle.  Tolerance:
the library's bars, 1e-13 log2 N (double), 1e-6 log2 N (float).
"""
import ctypes

import numpy as np
import pytest

from oracle import rel_l2

# shape, batch
CASES = [((8192,), 1), ((8192,), 3), ((16384,), 1), ((16384,), 3), ((1024, 2), 1), ((1024, 5), 3), ((2048, 3), 1),
         ((2048, 8), 2), ((2, 1024, 9), 1), ((3, 2048, 2), 2)]


def check(lib, oracle, dims, batch, put=lambda a: a, get=lambda a: a):
    n = int(np.prod(dims))
    bar = (1e-6 if lib.single else 1e-13) * np.log2(n)
    rng = np.random.default_rng(n + batch)
    x = (rng.uniform(-1, 1, (batch, n + 3)) + 1j * rng.uniform(-1, 1, (batch, n + 3))).astype(lib.cdt)
    with lib.mkaux("dft", dims) as a:
        for kind in ("dft", "invdft"):
            want = np.stack([oracle.nd(kind, r[:n].astype(complex).reshape(dims)).ravel() for r in x])
            y = put(np.zeros((batch, n + 1), lib.cdt))
            a.batched(kind, put(x), y, batch, n + 3, n + 1)
            assert rel_l2(get(y)[:, :n], want) <= bar, kind
            z = put(x.copy())
            a.batched(kind, z, z, batch, n + 3, n + 3)
            assert rel_l2(get(z)[:, :n], want) <= bar, kind + " in place"


@pytest.mark.parametrize("dims,batch", CASES)
@pytest.mark.parametrize("single", [False, True])
def test_emulated(emu_d, emu_f, oracle_d, dims, batch, single):
    lib = emu_f if single else emu_d
    count = lib.lib.nfft_emu_cluster_launches
    count.restype = ctypes.c_longlong
    before = count()
    check(lib, oracle_d, dims, batch)
    assert (count() > before) == (dims != ((8192,) if single else (16384,)))


@pytest.mark.gpu
@pytest.mark.parametrize("dims,batch", CASES)
@pytest.mark.parametrize("single", [False, True])
def test_gpu(lib_d, lib_f, oracle_d, dims, batch, single):
    import torch

    def get(t):
        torch.cuda.synchronize()
        return t.cpu().numpy()

    check(lib_f if single else lib_d, oracle_d, dims, batch, lambda a: torch.from_numpy(a).cuda(), get)
