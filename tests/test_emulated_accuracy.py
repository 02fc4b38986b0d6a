"""Relative L2 error of the transforms against extended precision, on the CPU
emulator: root tables, products of roots and butterflies are the kernels' own code.
A bound is the error of the general formulas on the same inputs (every root from the
tables, or the longest product chain of the 256-thread tiles), plus 1%.
"""
import numpy as np
import pytest

FAMILY = {"dft": "dft", "invdft": "dft", "realdft": "realdft", "invrealdft": "realdft", "dct2": "t2t3", "dct3": "t2t3",
          "dst2": "t2t3", "dst3": "t2t3", "dct4": "t4"}


def exact(kind, x):
    """Along the last axis, in the precision of x (unnormalized, FFTW's definitions)."""
    n = x.shape[-1]
    if kind == "dft":
        return np.fft.fft(x)
    if kind == "invdft":
        return np.fft.ifft(x) * (1 if n & (n - 1) else n)
    if kind == "realdft":
        return np.fft.rfft(x)
    if kind == "invrealdft":
        return np.fft.irfft(x) * (2 * n - 2)
    k = np.arange(n)
    turn = lambda num, den: np.exp(-1j * (np.longdouble("3.14159265358979323846264338327950288") * num / den))
    if kind == "dct2":
        return (np.fft.fft(np.concatenate([x, x[..., ::-1]], -1))[..., :n] * turn(k, 2 * n)).real
    if kind == "dst2":
        return exact("dct2", x * (1 - 2 * (k % 2)))[..., ::-1]
    if kind == "dct3":
        return np.fft.fft(x * np.where(k, 2, 1) * turn(k, 2 * n), 2 * n)[..., :n].real
    if kind == "dst3":
        return exact("dct3", x[..., ::-1]) * (1 - 2 * (k % 2))
    return (np.fft.fft(x * turn(k, 2 * n), 2 * n)[..., :n] * turn(2 * k + 1, 4 * n) * 2).real


def error(lib, kind, dims, batch):
    rng = np.random.default_rng(sum(dims))
    n = dims[-1]
    half = dims[:-1] + (n // 2 + 1,)
    ish, osh = (batch,) + (half if kind == "invrealdft" else dims), (batch,) + (half if kind == "realdft" else dims)
    x = rng.standard_normal(ish)
    if kind in ("dft", "invdft", "invrealdft"):
        x = x + 1j * rng.standard_normal(ish)
        if kind == "invrealdft":
            x[..., 0], x[..., -1] = x[..., 0].real, x[..., -1].real
        x = x.astype(lib.cdt)
    else:
        x = x.astype(lib.rdt)
    y = np.zeros(osh, lib.cdt if kind in ("dft", "invdft", "realdft") else lib.rdt)
    with lib.mkaux(FAMILY[kind], dims) as a:
        a.batched(kind, x, y, batch, x[0].size, y[0].size)
    want = x.astype(np.clongdouble if np.iscomplexobj(x) else np.longdouble)
    for axis in range(len(dims), 0, -1):
        want = np.moveaxis(exact(kind, np.moveaxis(want, axis, -1)), -1, axis)
    return float(np.sqrt((np.abs(y - want) ** 2).sum() / (np.abs(want) ** 2).sum()))


# kind, dims, batch: the general formulas' error in double and in float
BOUNDS = [
    # sub-stages of radix 8
    ("dft", (128,), 256, 2.406e-16, 1.225e-07),
    ("dft", (512,), 64, 2.732e-16, 1.382e-07),
    ("dft", (2048,), 16, 4.187e-16, 2.304e-07),
    ("dft", (8192,), 4, 4.428e-16, 2.432e-07),
    ("dft", (16384,), 2, 4.977e-16, 2.710e-07),
    ("realdft", (256,), 128, 2.572e-16, 1.310e-07),
    ("dct2", (1024,), 32, 3.126e-16, 1.554e-07),
    ("dft", (512, 32), 1, 3.080e-16, 1.604e-07),
    # input repack of DCT-3 / DST-3 and invrealdft
    ("dct3", (8192,), 4, 5.345e-16, 3.069e-07),
    ("dct3", (16384,), 2, 4.726e-16, 2.540e-07),
    ("dst3", (32768,), 1, 5.211e-16, 2.823e-07),
    ("invrealdft", (16384,), 2, 4.557e-16, 2.467e-07),
    # output unpack of realdft and DCT-2 / DST-2, whole lines
    ("realdft", (2048,), 16, 3.941e-16, 2.191e-07),
    ("realdft", (4096,), 8, 4.302e-16, 2.414e-07),
    ("dct2", (2048,), 16, 4.083e-16, 2.339e-07),
    ("dct2", (4096,), 8, 4.632e-16, 2.557e-07),
    ("dst2", (4096,), 8, 4.616e-16, 2.548e-07),
    # real-to-real transforms along strided axes; second twiddle of the multi-pass repack
    ("dct2", (64, 32), 8, 2.610e-16, 1.455e-07),
    ("dst2", (32, 32), 8, 2.529e-16, 1.422e-07),
    ("dct3", (256, 32), 4, 2.814e-16, 1.513e-07),
    ("dct3", (2048, 32), 1, 3.047e-16, 1.682e-07),
    ("dst3", (512, 32), 2, 2.863e-16, 1.577e-07),
    ("dct4", (1024, 32), 1, 5.721e-16, 1.578e-07),
    ("dct3", (131072,), 1, 6.411e-16, 3.640e-07),
    # Bluestein in one tile, padded to 2^13
    ("dft", (2049,), 7, 4.317e-16, 2.458e-07),
    ("dft", (2100,), 7, 4.386e-16, 2.510e-07),
    ("invdft", (2500,), 6, 4.993e-16, 2.777e-07),
    ("dft", (3000,), 5, 5.059e-16, 2.830e-07),
    ("dft", (4095,), 4, 5.758e-16, 3.296e-07),
]


@pytest.mark.parametrize("kind,dims,batch,double,single", BOUNDS)
def test_error(emu_d, emu_f, kind, dims, batch, double, single):
    assert error(emu_d, kind, dims, batch) <= 1.01 * double
    assert error(emu_f, kind, dims, batch) <= 1.01 * single
