"""Work buffers that fitted into a CTA's shared memory (or, for the TF32 sweep, twice into an SM's) when
the kernels had no operand tables, no channel lists and no table of buffers there still do: those are
paid for by buffers that are no longer needed.  The former sizes are restated here; the present ones
come from the kernels' own layout functions, compiled for the host."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from mpsqmc_b200 import build

CTA, SM, RESERVED = 232448, 233472, 1024  # B200: opt-in bytes of a CTA, of an SM, the driver's share per CTA


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("layout") / "liblayout.so")
    subprocess.run([nvcc, *build.NVCC_FLAGS, "-I", build.CSRC, os.path.join(ROOT, "tests", "cpp", "layout.cu"), "-o", out],
                   check=True, capture_output=True)
    f = C.CDLL(out).layout_bytes
    f.restype = C.c_long
    return f


def r4(n):
    return (n + 3) // 4 * 4


def padld(n):
    p = r4(n)
    return p + 4 if p % 8 == 0 else p


def former(kind, L, A, B, G):
    pa, pb, pq = padld(max(A, B)), padld(B), padld(2 * B)
    small = 16 * 8 + 2 * r4(B) + 56 + r4(G if kind < 2 else 1) + r4((L + 2) // 2) + r4(L) + 4
    env, site = pa * B, pb * B
    matrix = 8 * env + 4 * site  # Lenv, two products, four branches, one more; two site tensors of two blocks
    if kind == 0:
        matrix += pq * B + site  # Householder panel, R
    return 8 * small + (4 if kind == 1 else 8) * matrix


@pytest.mark.parametrize("L", [10, 64, 400])
def test_what_fitted_on_chip_still_does(layout, L):
    checked = 0
    for A in [*range(2, 130, 3), 160, 256, 400, 1000]:
        for B in [*range(2, min(A, 128) + 1, 2 if A < 100 else 5)]:
            for kind in range(3):
                was, now = former(kind, L, A, B, 240), layout(kind, L, A, B, 240)
                if was <= CTA:
                    assert now <= CTA, (kind, A, B, was, now)
                    checked += was > CTA - 30000
                if kind == 1 and 2 * (was + RESERVED) <= SM:
                    assert 2 * (now + RESERVED) <= SM, (kind, A, B, was, now)
    assert checked > 20
