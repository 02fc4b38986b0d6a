"""Which kernel a call takes, by the CPU emulator's launch counters: the tests of the
specialized kernels' values would pass on the general pass too.  And the cluster pass
as the first and last of a strided axis's two passes, against numpy in double (bars:
1e-13 log2 N double, 1e-6 log2 N float).
"""
import ctypes

import numpy as np
import pytest


def launches(lib):
    out = {"all": lib.launch_count()}
    for k in ("lean", "blue", "cluster"):
        f = getattr(lib.lib, f"nfft_emu_{k}_launches")
        f.restype = ctypes.c_longlong
        out[k] = f()
    return out


def taken(lib, family, kind, dims):
    n = int(np.prod(dims))
    x = np.ones(n, lib.cdt if family == "dft" else lib.rdt)
    y = np.zeros_like(x)
    with lib.mkaux(family, dims) as a:
        before = launches(lib)
        a.batched(kind, x, y, 1, n, n)
    return {k: v - before[k] for k, v in launches(lib).items()}


@pytest.mark.parametrize("single", [False, True])
def test_bluestein_tile(emu_d, emu_f, single):
    lib = emu_f if single else emu_d
    for n in (5, 17, 100, 1000, 2049, 4095):
        assert taken(lib, "dft", "dft", [n])["blue"] == 1, n
        assert taken(lib, "dft", "invdft", [n])["all"] == 1, n
    assert taken(lib, "dft", "dft", [3])["blue"] == 0
    assert taken(lib, "dft", "dft", [4097])["blue"] == 0


@pytest.mark.parametrize("single", [False, True])
def test_strided_real_to_real(emu_d, emu_f, single):
    lib = emu_f if single else emu_d
    for family, kinds in (("t2t3", ("dct2", "dct3", "dst2", "dst3")), ("t4", ("dct4", "dst4"))):
        for kind in kinds:
            for n in (32, 256, 2048):
                got = taken(lib, family, kind, [n, 32])
                assert (got["all"], got["lean"]) == (2, 2), (kind, n)


@pytest.mark.parametrize("single", [False, True])
def test_repack_of_several_passes(emu_d, emu_f, single):
    lib = emu_f if single else emu_d
    for kind in ("dct3", "dst3"):
        got = taken(lib, "t2t3", kind, [32768])
        assert (got["all"], got["lean"]) == (2, 2), kind


@pytest.mark.parametrize("n,single", [(1 << 20, False), (1 << 19, True)])
def test_cluster_passes_of_a_strided_axis(emu_d, emu_f, n, single):
    lib = emu_f if single else emu_d
    rng = np.random.default_rng(3)
    x = (rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2))).astype(lib.cdt)
    y = np.zeros_like(x)
    with lib.mkaux("dft", [n, 2]) as a:
        before = launches(lib)["cluster"]
        a.batched("dft", x, y, 1, 2 * n, 2 * n)
        assert launches(lib)["cluster"] - before == (1 if single else 2)
    want = np.fft.fft2(x.astype(complex))
    assert np.linalg.norm(y - want) / np.linalg.norm(want) <= (1e-6 if single else 1e-13) * 20
