"""What a call on another stream than its aux's previous call waits for: that call,
whose end is marked when it is made, and nothing else.  So it neither waits for what
the caller queued behind the call nor touches the previous call's stream, on which
work may be illegal by then.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

LEGACY_LINES, N = 8, 1024


def setup(lib):
    import torch
    x = torch.randn(LEGACY_LINES, N, dtype=torch.complex64 if lib.single else torch.complex128, device="cuda")
    return x, torch.zeros_like(x), torch.zeros_like(x)


@pytest.mark.parametrize("single", [False, True])
def test_unrelated_work_is_left_alone(lib_d, lib_f, single):
    import torch
    lib = lib_f if single else lib_d
    x, y, z = setup(lib)
    side = torch.cuda.Stream()
    with lib.mkaux("dft", [N]) as aux:
        for _ in range(3):
            try:
                lib.set_stream(None)
                aux.batched("dft", x, y, LEGACY_LINES, N, N)
                torch.cuda._sleep(300_000_000)   # 0.15 s or more behind the call
                behind = torch.cuda.Event()
                behind.record()
                lib.set_stream(side)
                aux.batched("dft", x, z, LEGACY_LINES, N, N)
                side.synchronize()
                assert not behind.query(), "the side stream's call waited for the work behind the previous call"
            finally:
                lib.set_stream(None)
                torch.cuda.synchronize()
            assert torch.equal(y, z)


@pytest.mark.parametrize("single", [False, True])
def test_a_blocking_stream_under_capture(lib_d, lib_f, single):
    import torch
    lib = lib_f if single else lib_d
    x, y, z = setup(lib)
    rt = ctypes.CDLL("libcudart.so.12")
    V = ctypes.c_void_p
    side, blocking, graph = torch.cuda.Stream(), V(), V()
    with lib.mkaux("dft", [N]) as aux:
        aux.batched("dft", x, y, LEGACY_LINES, N, N)
        lib.set_stream(side)
        aux.batched("dft", x, z, LEGACY_LINES, N, N)
        lib.set_stream(None)
        aux.batched("dft", x, y, LEGACY_LINES, N, N)
        torch.cuda.synchronize()
        z.zero_()
        torch.cuda.synchronize()
        assert rt.cudaStreamCreate(ctypes.byref(blocking)) == 0
        try:
            assert rt.cudaStreamBeginCapture(blocking, 2) == 0   # relaxed
            lib.set_stream(side)
            try:
                aux.batched("dft", x, z, LEGACY_LINES, N, N)
            finally:
                ended = rt.cudaStreamEndCapture(blocking, ctypes.byref(graph))
            assert ended == 0, "the capture was invalidated"
            side.synchronize()
            assert torch.equal(y, z)
        finally:
            lib.set_stream(None)
            if graph:
                rt.cudaGraphDestroy(graph)
            rt.cudaStreamDestroy(blocking)
