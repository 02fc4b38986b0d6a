"""Real-to-real transforms along a strided axis in one pass (whole lines in column
tiles): every length of the kernels' list at the axis, line counts that are no
multiple of a tile, padded distances, in place, adjoints; on the CPU emulator
(bounds-checked) and on the GPU, against the oracle.  Tolerance: the library's
bars, 1e-13 log2 N (double), 1e-6 log2 N (float), N the size of the plane.
"""
import numpy as np
import pytest

from oracle import rel_l2

SHAPES = [(32, 8), (64, 2), (128, 32), (256, 4), (512, 16), (1024, 2), (2048, 4), (32, 32, 2), (4, 64, 8)]
KINDS = [("t2t3", k) for k in ("dct2", "dst2", "dct3", "dst3")] + [("t4", "dct4"), ("t4", "dst4")]


def check(lib, oracle, dims, batch, put=lambda a: a, get=lambda a: a):
    n = int(np.prod(dims))
    bar = (1e-6 if lib.single else 1e-13) * np.log2(n)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (batch, n + 3)).astype(lib.rdt)
    for fam, kind in KINDS:
        want = np.stack([oracle.nd(kind, r[:n].astype(float).reshape(dims)).ravel() for r in x])
        with lib.mkaux(fam, dims) as a:
            y = put(np.zeros((batch, n + 1), lib.rdt))
            a.batched(kind, put(x), y, batch, n + 3, n + 1)
            assert rel_l2(get(y)[:, :n], want) <= bar, kind
            z = put(x.copy())
            a.batched(kind, z, z, batch, n + 3, n + 3)
            assert rel_l2(get(z)[:, :n], want) <= bar, kind + " in place"
            # <g, A x> = <A^T g, x>
            g = put(np.ascontiguousarray(x[:, ::-1]))
            gx = put(np.zeros((batch, n + 1), lib.rdt))
            a.vjp_batched(kind, g, gx, batch, n + 3, n + 1)
            lhs = np.sum(get(g)[:, :n].astype(float) * want)
            rhs = np.sum(get(gx)[:, :n].astype(float) * x[:, :n])
            scale = np.linalg.norm(get(g)[:, :n].astype(float)) * np.linalg.norm(want)
            assert abs(lhs - rhs) <= bar * scale, kind + " adjoint"


@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("single", [False, True])
def test_emulated(emu_d, emu_f, oracle_d, dims, single):
    check(emu_f if single else emu_d, oracle_d, dims, 3)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", SHAPES)
@pytest.mark.parametrize("single", [False, True])
def test_gpu(lib_d, lib_f, oracle_d, dims, single):
    import torch

    def get(t):
        torch.cuda.synchronize()
        return t.cpu().numpy()

    check(lib_f if single else lib_d, oracle_d, dims, 3, lambda a: torch.from_numpy(a).cuda(), get)
