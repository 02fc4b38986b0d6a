"""Chains of calls on grids at the lines of the rule that picks dependent or plain
launches (halves, two thirds, four fifths and all of the chip's CTA places, and beside
them): each call reads what the one before wrote, and a chain gives bit for bit what
the same calls give with a synchronization after each.
"""
import pytest

pytestmark = pytest.mark.gpu

# family, forward, inverse, length, transforms per CTA (2048-point tiles)
CHAINS = [("dft", "dft", "invdft", 1024, 2), ("realdft", "realdft", "invrealdft", 64, 64), ("t2t3", "dct2", "dct3", 512, 8),
          ("dft", "dft", "invdft", 1000, 1)]


@pytest.mark.parametrize("single", [False, True])
@pytest.mark.parametrize("family,fwd,inv,n,per", CHAINS)
def test_chain(lib_d, lib_f, single, family, fwd, inv, n, per):
    import torch
    lib = lib_f if single else lib_d
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    places = sms * (8 if single else 4)
    rdt, cdt = (torch.float32, torch.complex64) if single else (torch.float64, torch.complex128)
    half = n // 2 + 1 if family == "realdft" else n
    for ctas in (sms - 1, places // 2, places // 2 + 1, 2 * places // 3, 4 * places // 5, 4 * places // 5 + 1, places + 1):
        b = ctas * per
        x = torch.randn(b, n, dtype=cdt if family == "dft" else rdt, device="cuda")
        with lib.mkaux(family, [n]) as aux:
            def chain(wait):
                u = x.clone()
                v = torch.zeros(b, half, dtype=cdt if family != "t2t3" else rdt, device="cuda")
                for _ in range(4):
                    aux.batched(fwd, u, v, b, n, half)
                    if wait:
                        torch.cuda.synchronize()
                    aux.batched(inv, v, u, b, half, n)
                    if wait:
                        torch.cuda.synchronize()
                return u, v
            got, want = chain(False), chain(True)
            assert torch.isfinite(torch.view_as_real(want[0]) if want[0].is_complex() else want[0]).all()
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), ctas
