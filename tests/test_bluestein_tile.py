"""Single-tile Bluestein kernels: the shortest and longest length of every padded
size, batches that end inside a tile, padded distances, both directions, in
place; on the CPU emulator (bounds-checked) and on the GPU, against the oracle.
Tolerance: the library's bars, 1e-13 log2 N (double) and 1e-6 log2 N (float).
"""
import math

import numpy as np
import pytest

from oracle import rel_l2

# (length, transforms): M = 16 .. 8192, tiles of 2048 points and one line above
CASES = [(5, 257), (7, 3), (9, 130), (15, 1), (17, 33), (31, 65), (33, 17), (63, 2), (65, 9), (127, 8), (129, 5),
         (255, 4), (257, 3), (511, 1), (513, 3), (1000, 2), (1025, 1), (2047, 2), (2049, 1), (4095, 2)]


def check(lib, oracle, n, batch, put=lambda a: a, get=lambda a: a, device=False):
    bar = (1e-6 if lib.single else 1e-13) * math.log2(n)
    rng = np.random.default_rng(n)
    x = (rng.uniform(-1, 1, (batch, n + 3)) + 1j * rng.uniform(-1, 1, (batch, n + 3))).astype(lib.cdt)
    with lib.mkaux("dft", [n]) as a:
        for kind in ("dft", "invdft"):
            want = np.stack([oracle.transform(kind, r) for r in x[:, :n].astype(complex)])
            y = put(np.zeros((batch, n + 1), lib.cdt))
            a.batched(kind, put(x), y, batch, n + 3, n + 1)
            assert rel_l2(get(y)[:, :n], want) <= bar, kind
            z = put(x.copy())
            a.batched(kind, z, z, batch, n + 3, n + 3)
            assert rel_l2(get(z)[:, :n], want) <= bar, kind + " in place"
            if device:   # host arrays are staged whole
                assert np.array_equal(get(z)[:, n:], x[:, n:]), "stores outside the lines"


@pytest.mark.parametrize("n,batch", CASES)
@pytest.mark.parametrize("single", [False, True])
def test_emulated(emu_d, emu_f, oracle_d, n, batch, single):
    check(emu_f if single else emu_d, oracle_d, n, batch)


@pytest.mark.gpu
@pytest.mark.parametrize("n,batch", CASES)
@pytest.mark.parametrize("single", [False, True])
def test_gpu(lib_d, lib_f, oracle_d, n, batch, single):
    import torch

    def get(t):
        torch.cuda.synchronize()
        return t.cpu().numpy()

    check(lib_f if single else lib_d, oracle_d, n, batch, lambda a: torch.from_numpy(a).cuda(), get, True)


# ---- the same tiles as branches of the ragged queue ---------------------------
def check_queue(lib, oracle, put=lambda a: a, get=lambda a: a):
    rng = np.random.default_rng(5)
    ns = [5, 7, 9, 15, 17, 33, 63, 65, 127, 129, 255, 257, 511, 513, 1000, 1023, 1025, 2047]
    kinds = [k for n in ns for k in ("dft", "invdft", "realdft", "dct2", "realdft")]
    lens = [n for n in ns for _ in range(5)]
    with lib.mkbatch(kinds, lens) as b:
        x = rng.uniform(-1, 1, b.in_size).astype(lib.rdt)
        y = put(np.zeros(b.out_size, lib.rdt))
        b.execute(put(x), y)
        assert b.status() == 0
        y = get(y).astype(float)
    xi = yo = 0
    for kind, n in zip(kinds, lens):
        cplx = kind in ("dft", "invdft")
        ni, no = (2 * n, 2 * n) if cplx else (n, 2 * (n // 2 + 1) if kind == "realdft" else n)
        v = x[xi:xi + ni].astype(float)
        if cplx:
            want = oracle.transform(kind, v[0::2] + 1j * v[1::2])
        elif kind == "realdft":
            want = oracle.transform("dft", v.astype(complex))[:n // 2 + 1]
        else:
            q = np.arange(n)
            w = np.concatenate([v[0::2], v[1::2][::-1]]).astype(complex)
            want = 2 * (np.exp(-0.5j * np.pi * q / n) * oracle.transform("dft", w)).real
        got = y[yo:yo + no]
        got = got[0::2] + 1j * got[1::2] if kind != "dct2" else got
        assert rel_l2(got, want) <= (1e-6 if lib.single else 1e-13) * math.log2(n), (kind, n)
        xi += ni + (ni & 1)
        yo += no + (no & 1)


@pytest.mark.parametrize("single", [False, True])
def test_queue_emulated(emu_d, emu_f, oracle_d, single):
    check_queue(emu_f if single else emu_d, oracle_d)


@pytest.mark.gpu
@pytest.mark.parametrize("single", [False, True])
def test_queue_gpu(lib_d, lib_f, oracle_d, single):
    import torch

    check_queue(lib_f if single else lib_d, oracle_d, lambda a: torch.from_numpy(a).cuda(), lambda t: t.cpu().numpy())
