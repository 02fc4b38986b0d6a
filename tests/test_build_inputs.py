"""What a build of the libraries needs besides a C++17 compiler: the CUDA runtime,
driver and half-precision headers.  Headers that pull in the toolkit's C++ template
libraries are left out, so that a checkout builds wherever nvcc alone is installed;
and a file that does not compile ends the build with the compiler's message.
"""
import os
import re
import time

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "notorious-fft_b200", "csrc")


def test_toolkit_headers():
    used = set()
    for name in os.listdir(CSRC):
        with open(os.path.join(CSRC, name)) as f:
            used |= set(re.findall(r"^\s*#\s*include\s*<([^>]+)>", f.read(), flags=re.M))
    templates = ("cooperative_groups", "cub/", "cuda/", "cute/", "cutlass/", "nv/", "thrust/")
    assert not [h for h in used if h.startswith(templates)]


def test_first_error_ends_the_build(monkeypatch):
    import build

    started = []

    def compile_one(src, prec, extra, verbose):
        started.append(src)
        if len(started) == 1:
            raise RuntimeError(f"nvcc failed for {src}")
        time.sleep(0.2)
        return src

    monkeypatch.setattr(build, "compile_one", compile_one)
    with pytest.raises(RuntimeError, match="nvcc failed for"):
        build.build(jobs=1)
    assert len(started) < len(build.SOURCES)
