"""The paired input repack of DCT-3 / DST-3 and the inverse real transform, in
row tiles (one pass) and mirrored tiles (first of several passes): every pass
radix of the kernels' list, odd batches, padded distances, and the adjoints that
run through it, on the CPU emulator (bounds-checked) and on the GPU, against the
oracle.  Tolerance: the library's bars, 1e-13 log2 N (double), 1e-6 log2 N (float).
"""
import numpy as np
import pytest

from oracle import rel_l2

SIZES = [32, 64, 256, 1024, 4096, 8192, 16384, 1 << 15, 1 << 16]
LARGE = [1 << 17, 1 << 19, 1 << 20, 1 << 22]   # first passes of radix 2^8 .. 2^9, three passes


def check(lib, oracle, n, batch, put=lambda a: a, get=lambda a: a):
    bar = (1e-6 if lib.single else 1e-13) * np.log2(n)
    rng = np.random.default_rng(n)
    h = n // 2 + 1
    x = rng.uniform(-1, 1, (batch, n + 1)).astype(lib.rdt)
    z = (rng.uniform(-1, 1, (batch, h + 2)) + 1j * rng.uniform(-1, 1, (batch, h + 2))).astype(lib.cdt)
    xs, zs = x[:, :n].astype(float), z[:, :h].astype(complex)
    sign = 1.0 - 2.0 * (np.arange(n) % 2)
    rows = lambda kind, a: np.stack([oracle.transform(kind, r) for r in a])  # noqa: E731
    want = {"dct3": rows("dct3", xs), "dst3": rows("dst3", xs)}
    with lib.mkaux("t2t3", [n]) as a:
        for kind in want:
            y = put(np.zeros((batch, n + 3), lib.rdt))
            a.batched(kind, put(x), y, batch, n + 1, n + 3)
            assert rel_l2(get(y)[:, :n], want[kind]) <= bar, kind
        adj = {"dct2": want["dct3"] + xs[:, :1], "dst2": want["dst3"] + sign * xs[:, -1:]}
        for kind in adj:
            y = put(np.zeros((batch, n + 3), lib.rdt))
            a.vjp_batched(kind, put(x), y, batch, n + 1, n + 3)
            assert rel_l2(get(y)[:, :n], adj[kind]) <= bar, kind + " adjoint"
    with lib.mkaux("realdft", [n]) as a:
        y = put(np.zeros((batch, n + 3), lib.rdt))
        a.batched("invrealdft", put(z), y, batch, h + 2, n + 3)
        assert rel_l2(get(y)[:, :n], np.stack([oracle.invrealdft(r, n) for r in zs])) <= bar
        a.vjp_batched("realdft", put(z), y, batch, h + 2, n + 3)
        half = zs.copy()
        half[:, 1:-1] *= 0.5
        assert rel_l2(get(y)[:, :n], np.stack([oracle.invrealdft(r, n) for r in half])) <= bar


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("single", [False, True])
def test_emulated(emu_d, emu_f, oracle_d, n, single):
    check(emu_f if single else emu_d, oracle_d, n, 3 if n > 1024 else 9)


@pytest.mark.gpu
@pytest.mark.parametrize("n", SIZES + LARGE)
@pytest.mark.parametrize("single", [False, True])
def test_gpu(lib_d, lib_f, oracle_d, n, single):
    import torch

    def get(t):
        torch.cuda.synchronize()
        return t.cpu().numpy()

    check(lib_f if single else lib_d, oracle_d, n, 3 if n > 1024 else 9, lambda a: torch.from_numpy(a).cuda(), get)
