"""Timed cases of the FFT library: what its users have it do, on device memory.

A case is one program step through the public binding (`notorious_fft.Library`):
plans are made and buffers allocated in `prepare`, `run` makes the library calls.
Host-memory calls are left out on purpose: the PCIe link, not this library's
kernels, is what such a call takes its time on.

Keys of a case
  family  "dft"     complex transform of shape `dims` (any length; lengths that
                    are not powers of two run by Bluestein's algorithm)
          "real"    realdft, with `both` then invrealdft of its output
          "t2t3"    dct2 (dst2), with `both` then dct3 (dst3) of its output
          "t4"      dct4 (dst4)
          "ragged"  one batch of `count` transforms of mixed kinds and lengths
          "grad"    a differentiated step: 2-D realdft and 1-D dct2, and the
                    adjoints of both on their cotangents
  dims    "512x512": the transform's shape;  batch: transforms per call
  prec    "f64" or "f32" (the double and the float library)
  both    the forward transform and the inverse of its output
  dst     the sine variant of the real-to-real families
  split   the float library's split tensor-core form
"""
import math
import os
import random
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "notorious-fft_b200"))

import notorious_fft as nf  # noqa: E402


def listed():
    return [
        # one transform of one line: a call inside somebody's loop, all latency
        dict(name="c2c_f64_1024", family="dft", prec="f64", dims="1024", batch=1, both=False),
        # filtering of short lines: there and back, 256 lines of 4096 points
        dict(name="c2c_f64_4096x256", family="dft", prec="f64", dims="4096", batch=256, both=True),
        # the headline workload: 4096 lines of 65536 points, there and back
        dict(name="c2c_f64_65536x4096", family="dft", prec="f64", dims="65536", batch=4096, both=True),
        # the same lines in single precision through the split tensor-core form
        dict(name="c2c_f32_split_65536x1024", family="dft", prec="f32", dims="65536", batch=1024, both=True, split=True),
        # spectra of single-precision records, an odd number of them
        dict(name="c2c_f32_16384x1001", family="dft", prec="f32", dims="16384", batch=1001, both=False),
        # long real signals to their half spectrum and back
        dict(name="real_f64_1048576x16", family="real", prec="f64", dims="1048576", batch=16, both=True),
        # a spectral solver's cosine transform along lines, and its inverse
        dict(name="dct_f64_8192x512", family="t2t3", prec="f64", dims="8192", batch=512, both=True),
        # one image-sized plane
        dict(name="c2c_f64_2048x2048", family="dft", prec="f64", dims="2048x2048", batch=1, both=False),
        # lines of a length that is not a power of two
        dict(name="c2c_f64_1000x2000", family="dft", prec="f64", dims="1000", batch=2000, both=False),
        # a long prime length
        dict(name="c2c_f64_1000003x4", family="dft", prec="f64", dims="1000003", batch=4, both=False),
        # a service's queue: many transforms of uneven lengths and kinds at once
        dict(name="ragged_f64_1000", family="ragged", prec="f64", count=1000, nmax=262144, sizes=7),
        # a differentiable loss on a batch of images
        dict(name="grad_f32_512x512x64", family="grad", prec="f32", dims="512x512", batch=64),
    ]


def _odd(rng, v):
    """A count near v that is odd half of the time."""
    v = max(1, int(round(v)))
    return v if v < 3 or rng.random() < 0.5 else v | 1


def _total(rng, lo, hi):
    return 2.0 ** rng.uniform(math.log2(lo), math.log2(hi))


def draw(rng):
    prec = "f64" if rng.random() < 0.6 else "f32"
    pick = rng.random()
    if pick < 0.30:      # lines of a power of two
        n = 1 << rng.randint(4, 20)
        batch = _odd(rng, _total(rng, max(n, 1 << 10), 1 << 26) / n)
        c = dict(family="dft", prec=prec, dims=str(n), batch=batch, both=rng.random() < 0.5)
        if prec == "f32" and rng.random() < 0.3:
            c["split"] = True
        return c
    if pick < 0.42:      # planes and volumes
        if rng.random() < 0.6:
            dims = [1 << rng.randint(6, 11) for _ in range(2)]
        else:
            dims = [1 << rng.randint(4, 8) for _ in range(3)]
        size = math.prod(dims)
        batch = _odd(rng, _total(rng, size, 1 << 25) / size)
        return dict(family="dft", prec=prec, dims="x".join(map(str, dims)), batch=batch, both=rng.random() < 0.3)
    if pick < 0.58:      # real lines and planes
        if rng.random() < 0.7:
            dims = [1 << rng.randint(5, 20)]
        else:
            dims = [1 << rng.randint(6, 11) for _ in range(2)]
        size = math.prod(dims)
        batch = _odd(rng, _total(rng, max(size, 1 << 11), 1 << 26) / size)
        return dict(family="real", prec=prec, dims="x".join(map(str, dims)), batch=batch, both=rng.random() < 0.6)
    if pick < 0.72:      # cosine and sine transforms
        if rng.random() < 0.75:
            dims = [1 << rng.randint(5, 18)]
        else:
            dims = [1 << rng.randint(5, 10) for _ in range(2)]
        size = math.prod(dims)
        batch = _odd(rng, _total(rng, max(size, 1 << 11), 1 << 25) / size)
        c = dict(family="t2t3" if rng.random() < 0.7 else "t4", prec=prec, dims="x".join(map(str, dims)), batch=batch,
                 dst=rng.random() < 0.4)
        if c["family"] == "t2t3":
            c["both"] = rng.random() < 0.6
        return c
    if pick < 0.86:      # lengths that are not powers of two
        n = int(_total(rng, 17, 1 << 20))
        if rng.random() < 0.4 and n > 100:   # round numbers are common
            n = int(float("%.1e" % n))
        if n & (n - 1) == 0:
            n += 1
        batch = _odd(rng, _total(rng, max(n, 1 << 10), 1 << 23) / n)
        return dict(family="dft", prec=prec, dims=str(n), batch=batch, both=rng.random() < 0.3)
    if pick < 0.93:      # uneven batches
        return dict(family="ragged", prec=prec, count=_odd(rng, _total(rng, 60, 1500)), nmax=1 << rng.randint(10, 18),
                    sizes=rng.randint(0, 1 << 20))
    dims = [1 << rng.randint(6, 10) for _ in range(2)]
    size = math.prod(dims)
    return dict(family="grad", prec=prec, dims="x".join(map(str, dims)),
                batch=_odd(rng, _total(rng, size, 1 << 24) / size))


# ---- shapes -------------------------------------------------------------------
def _dims(case):
    return [int(v) for v in case["dims"].split("x")]


def _types(case):
    return (torch.float64, torch.complex128) if case["prec"] == "f64" else (torch.float32, torch.complex64)


def _half(dims):
    return dims[:-1] + [dims[-1] // 2 + 1]


def _prime(n):
    if n < 4 or n % 2 == 0:
        return n in (2, 3)
    return all(n % p for p in range(3, math.isqrt(n) + 1, 2))


def _ragged_list(case):
    """Kinds and lengths: half complex, 30% real, 20% cosine; lengths spread over
    their logarithm, a fifth of them no powers of two, half of those prime."""
    rng = random.Random(case["sizes"])
    kinds, ns = [], []
    for _ in range(case["count"]):
        u = rng.random()
        kinds.append("dft" if u < 0.5 else "realdft" if u < 0.8 else "dct2")
        n = max(16, int(_total(rng, 16, case["nmax"])))
        v = rng.random()
        if v < 0.8:
            n = 1 << int(round(math.log2(n)))
        elif v < 0.9:
            while not _prime(n):
                n += 1
        else:
            while n & (n - 1) == 0 or _prime(n):
                n += 1
        ns.append(n)
    return kinds, ns


def _ragged_reals(kind, n):
    """Reals read and written by one transform."""
    return (2 * n if kind == "dft" else n), (2 * n if kind == "dft" else 2 * (n // 2 + 1) if kind == "realdft" else n)


# ---- inputs -------------------------------------------------------------------
def _randn(gen, shape, dtype):
    return torch.randn(shape, generator=gen, dtype=dtype, device="cuda")


def _inputs(case, seed):
    """The case's inputs, from the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rdt, cdt = _types(case)
    fam = case["family"]
    if fam == "ragged":
        with_len = sum(_ragged_reals(k, n)[0] + (_ragged_reals(k, n)[0] & 1) for k, n in zip(*_ragged_list(case)))
        return torch.rand((with_len,), generator=gen, dtype=rdt, device="cuda") * 2 - 1
    shape = [case["batch"]] + _dims(case)
    if fam == "dft":
        return _randn(gen, shape, cdt)
    if fam == "grad":
        return dict(x=_randn(gen, shape, rdt), gz=_randn(gen, _half(shape), cdt),
                    m=_randn(gen, shape[:2], rdt), gm=_randn(gen, shape[:2], rdt))
    return _randn(gen, shape, rdt)


def prepare(case, seed):
    lib = nf.load(single=case["prec"] == "f32")
    rdt, cdt = _types(case)
    fam = case["family"]
    x = _inputs(case, seed)
    st = dict(case=case, lib=lib, x=x)
    if fam == "ragged":
        kinds, ns = _ragged_list(case)
        st["plan"] = lib.mkbatch(kinds, ns)
        st["y"] = torch.zeros((st["plan"].out_size,), dtype=rdt, device="cuda")
        return st
    dims, b = _dims(case), case["batch"]
    if fam == "dft":
        st["plan"] = lib.mkaux("dft", dims)
        if case.get("split"):
            st["plan"].set_form(nf.FORM_SPLIT_TC)
        st["y"] = torch.empty_like(x)
    elif fam == "real":
        st["plan"] = lib.mkaux("realdft", dims)
        st["y"] = torch.empty([b] + _half(dims), dtype=cdt, device="cuda")
    elif fam in ("t2t3", "t4"):
        st["plan"] = lib.mkaux(fam, dims)
        st["y"] = torch.empty_like(x)
    else:
        st["plan"] = lib.mkaux("realdft", dims)
        st["lines"] = lib.mkaux("t2t3", [dims[0]])
        st["out"] = dict(z=torch.empty_like(x["gz"]), gx=torch.empty_like(x["x"]), d=torch.empty_like(x["m"]),
                         gd=torch.empty_like(x["m"]))
    if case.get("both"):
        st["z"] = torch.empty_like(x)
    return st


# ---- the calls ------------------------------------------------------------------
def _kinds(case):
    fam = case["family"]
    s = "s" if case.get("dst") else "c"
    fwd, inv = {"dft": ("dft", "invdft"), "real": ("realdft", "invrealdft"), "t2t3": (f"d{s}t2", f"d{s}t3"),
                "t4": (f"d{s}t4", None)}[fam]
    return fwd, (inv if case.get("both") else None)


def _call(plan, kind, x, y, b):
    if b == 1:
        plan(kind, x, y)
    else:
        plan.batched(kind, x, y, b, x.numel() // b, y.numel() // b)


def run(state):
    case = state["case"]
    if case["family"] == "ragged":
        state["plan"].execute(state["x"], state["y"])
        return state["y"]
    b = case["batch"]
    if case["family"] == "grad":
        i, o = state["x"], state["out"]
        full, half, line = i["x"].numel() // b, i["gz"].numel() // b, i["m"].shape[1]
        state["plan"].batched("realdft", i["x"], o["z"], b, full, half)
        state["lines"].batched("dct2", i["m"], o["d"], b, line, line)
        state["plan"].vjp_batched("realdft", i["gz"], o["gx"], b, half, full)
        state["lines"].vjp_batched("dct2", i["gm"], o["gd"], b, line, line)
        return o
    fwd, inv = _kinds(case)
    _call(state["plan"], fwd, state["x"], state["y"], b)
    if inv is None:
        return [state["y"]]
    _call(state["plan"], inv, state["y"], state["z"], b)
    return [state["y"], state["z"]]


# ---- work ---------------------------------------------------------------------
def _line_flops(n, real):
    return 5.0 * n * math.log2(max(n, 2)) * (0.5 if real else 1.0)


def work(case):
    r = 8 if case["prec"] == "f64" else 4
    fam = case["family"]
    if fam == "ragged":
        ks, ns = _ragged_list(case)
        return dict(bytes=r * sum(sum(_ragged_reals(k, n)) for k, n in zip(ks, ns)),
                    flops=sum(_line_flops(n, k != "dft") for k, n in zip(ks, ns)))
    dims, b = _dims(case), case["batch"]
    size = math.prod(dims)
    real = fam != "dft"
    flops = b * _line_flops(size, real)
    io = {"dft": 4 * size, "real": size + 2 * math.prod(_half(dims)), "t2t3": 2 * size, "t4": 2 * size,
          "grad": 2 * (size + 2 * math.prod(_half(dims)) + 2 * dims[0])}[fam]
    times = 2 if case.get("both") or fam == "grad" else 1
    return dict(bytes=b * r * io * (2 if case.get("both") else 1), flops=times * flops)


# ---- 64-bit values --------------------------------------------------------------
def _turn(num, den):
    """exp(-i pi num / den)."""
    a = num.double() * (math.pi / den)
    return torch.complex(torch.cos(a), -torch.sin(a))


def _r2r(x, kind, axis):
    """A cosine / sine transform (unnormalized, FFTW's definitions) along an axis."""
    x = x.movedim(axis, -1)
    n = x.shape[-1]
    k = torch.arange(n, device=x.device)
    sign = (1 - 2 * (k % 2)).double()
    if kind == "dct2":
        y = (torch.fft.fft(torch.cat([x, x.flip(-1)], -1))[..., :n] * _turn(k, 2 * n)).real
    elif kind == "dst2":
        y = _r2r(x * sign, "dct2", -1).flip(-1)
    elif kind == "dct3":
        w = torch.full((n,), 2.0, dtype=torch.float64, device=x.device)
        w[0] = 1.0
        y = torch.fft.fft(x * w * _turn(k, 2 * n), 2 * n)[..., :n].real
    elif kind == "dst3":
        y = _r2r(x.flip(-1), "dct3", -1) * sign
    else:
        t = torch.fft.fft(x * _turn(k, 2 * n), 2 * n)[..., :n] * _turn(2 * k + 1, 4 * n) * 2
        y = t.real if kind == "dct4" else -t.imag
    return y.movedim(-1, axis)


def _exact_1d(x, kind):
    if kind == "dft":
        return torch.view_as_real(torch.fft.fft(torch.view_as_complex(x.view(-1, 2)))).reshape(-1)
    if kind == "realdft":
        return torch.view_as_real(torch.fft.rfft(x)).reshape(-1)
    return _r2r(x, "dct2", -1)


def exact(case, seed):
    fam = case["family"]
    x = _inputs(case, seed)
    if fam == "ragged":
        x, outs = x.double(), []
        at = 0
        for k, n in zip(*_ragged_list(case)):
            ni = _ragged_reals(k, n)[0]
            v = _exact_1d(x[at:at + ni], k)
            outs.append(torch.nn.functional.pad(v, (0, v.numel() & 1)))
            at += ni + (ni & 1)
        y = torch.cat(outs)
        return y[:y.numel() - 1] if _last_odd(case) else y
    if fam == "grad":
        n2 = _dims(case)[1]
        g = x["gz"].to(torch.complex128)
        full = torch.nn.functional.pad(g, (0, n2 - g.shape[-1]))
        gm = x["gm"].double()
        return dict(z=torch.fft.rfft2(x["x"].double()), gx=torch.fft.ifft2(full, norm="forward").real,
                    d=_r2r(x["m"].double(), "dct2", -1),
                    gd=_r2r(gm, "dct3", -1) + gm[:, :1])
    axes = list(range(1, 1 + len(_dims(case))))
    fwd, inv = _kinds(case)
    if fam == "dft":
        x = x.to(torch.complex128)
        y = torch.fft.fftn(x, dim=axes)
        size = math.prod(_dims(case))
        back = x * (size if size & (size - 1) == 0 else 1)
    elif fam == "real":
        x = x.double()
        y = torch.fft.rfftn(x, dim=axes)
        back = x * math.prod(_dims(case))
    else:
        y = x.double()
        for a in axes:
            y = _r2r(y, fwd, a)
        back = None
        if inv:
            back = y
            for a in axes:
                back = _r2r(back, inv, a)
    return [y] if inv is None else [y, back]


def _last_odd(case):
    """Whether the last transform's output is of odd length: nothing pads it."""
    ks, ns = _ragged_list(case)
    return _ragged_reals(ks[-1], ns[-1])[1] & 1 == 1
