"""Consecutive kernels overlap (dependent launches): long chains of calls without a
synchronization, in place and through alternating buffers, at grid sizes from a
few CTAs to many waves, must give exactly what the same calls give one by one;
and a captured chain replays on new data.
"""
import pytest

pytestmark = pytest.mark.gpu

# (kind, inverse, length, batch): one CTA .. many waves; one, two and three passes
CHAINS = [("dft", "invdft", 64, 3), ("dft", "invdft", 4096, 115), ("dft", "invdft", 4096, 900),
          ("dft", "invdft", 1 << 16, 40), ("dft", "invdft", 1 << 19, 9), ("dft", "invdft", 1000, 77),
          ("dct2", "dct3", 4096, 230), ("dct2", "dct3", 1 << 15, 33), ("dct4", "dct4", 512, 64),
          ("dft", "invdft", 5213, 20)]


def buffers(lib, kind, n, batch):
    import torch
    real = torch.float32 if lib.single else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand((batch, n), generator=gen, dtype=real, device="cuda") - 0.5
    return torch.complex(x, x.flip(1)) if kind == "dft" else x


def chain(lib, aux, kind, inverse, bufs, n, batch, steps, wait):
    import torch
    a, b = bufs
    scale = 1.0 / n if n & (n - 1) == 0 and kind == "dft" else 1.0 if kind == "dft" else 1.0 / (2 * n)
    for k in range(steps):
        aux.batched(kind, a, b, batch, n, n)
        if wait:
            torch.cuda.synchronize()
        aux.batched(inverse, b, b, batch, n, n)      # in place
        if wait:
            torch.cuda.synchronize()
        if k % 3 == 2:
            b.mul_(scale ** 3)                       # another library's kernel in between
        a, b = b, a
    return a


@pytest.mark.parametrize("case", CHAINS, ids=lambda c: f"{c[0]}-{c[2]}x{c[3]}")
@pytest.mark.parametrize("single", [False, True])
def test_chain(lib_d, lib_f, case, single):
    import torch
    lib = lib_f if single else lib_d
    kind, inverse, n, batch = case
    x = buffers(lib, kind, n, batch)
    with lib.mkaux(kind, [n]) as aux:
        got = chain(lib, aux, kind, inverse, (x.clone(), torch.zeros_like(x)), n, batch, 9, wait=False)
        want = chain(lib, aux, kind, inverse, (x.clone(), torch.zeros_like(x)), n, batch, 9, wait=True)
        torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("single", [False, True])
def test_captured_chain(lib_d, lib_f, single):
    import torch
    lib = lib_f if single else lib_d
    n, batch = 1 << 16, 12
    x = buffers(lib, "dft", n, batch)
    y, z = torch.zeros_like(x), torch.zeros_like(x)
    with lib.mkaux("dft", [n]) as aux:
        aux.batched("dft", x, y, batch, n, n)        # plan scratch
        torch.cuda.synchronize()
        graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=stream):
            lib.set_stream(stream)
            aux.batched("dft", x, y, batch, n, n)
            aux.batched("invdft", y, z, batch, n, n)
            aux.batched("dft", z, z, batch, n, n)
        lib.set_stream(None)
        for k in range(3):
            x.mul_(-0.5)
            graph.replay()
            torch.cuda.synchronize()
            got = z.clone()
            aux.batched("dft", x, y, batch, n, n)
            aux.batched("invdft", y, z, batch, n, n)
            aux.batched("dft", z, z, batch, n, n)
            torch.cuda.synchronize()
            assert torch.equal(got, z), k
        del graph


@pytest.mark.parametrize("single", [False, True])
def test_alternating_streams(lib_d, lib_f, single):
    """One aux (and its scratch) on the default stream and on two others in turn,
    without a synchronization: every call waits for the one before."""
    import torch
    lib = lib_f if single else lib_d
    n, batch = 1 << 17, 24
    xs = [buffers(lib, "dft", n, batch) * (k + 1) for k in range(6)]
    ys = [torch.zeros_like(x) for x in xs]
    streams = [None, torch.cuda.Stream(), None, torch.cuda.Stream(), None]
    with lib.mkaux("dft", [n]) as aux:
        torch.cuda.synchronize()
        for rep in range(4):
            for k, (x, y) in enumerate(zip(xs, ys)):
                lib.set_stream(streams[(k + rep) % len(streams)])
                aux.batched("dft", x, y, batch, n, n)
        lib.set_stream(None)
        torch.cuda.synchronize()
        want = torch.zeros_like(xs[0])
        for x, y in zip(xs, ys):
            aux.batched("dft", x, want, batch, n, n)
            torch.cuda.synchronize()
            assert torch.equal(y, want)
