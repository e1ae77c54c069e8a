"""The grid point that a coupling samples (sample_grid) against the serial CDF scan it stands for
(MPSQMC2.cpp:577-588): first point whose cumulative PDF exceeds u, point 0 where the sum of the PDF is
zero (the comparison with a NaN ends the reference's scan at once), never a point of
probability zero.  Uniforms sit in the rounding gaps between a lane's run and the next lane's, on
the cumulative sums themselves and at random.  The sampled point's cumulative sum may miss u by the
rounding of a sum of G terms, G 2^-52."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from mpsqmc_b200 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scan(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("scan") / "libsample_scan.so")
    subprocess.run([nvcc, *build.NVCC_FLAGS, "-I", build.CSRC, os.path.join(ROOT, "tests", "cpp", "sample_scan.cu"),
                    "-o", out], check=True, capture_output=True)
    lib = C.CDLL(out)

    def run(grids, u, ov, threads):
        n, G = grids.shape[:2]
        grids, u = np.ascontiguousarray(grids), np.ascontiguousarray(u)
        index, factor = np.empty(n, np.int32), np.empty(n)
        ptr = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
        assert lib.sample_scan(n, G, threads, C.c_double(ov), ptr(grids), ptr(u), ptr(index), ptr(factor)) == 0
        return index, factor
    return run


def lanes(pdf):
    """A warp's sums over runs of the grid: (running sums of each lane, sum in front of each lane, total)."""
    per = (len(pdf) + 31) // 32
    run = np.zeros((32, per))
    run.reshape(-1)[:len(pdf)] = pdf
    mine = np.zeros(32)
    for i in range(per):
        mine = mine + run[:, i]
    cum, o = mine.copy(), 1
    while o < 32:
        cum[o:] = cum[o:] + cum[:-o].copy()
        o *= 2
    first = np.concatenate([[0.0], cum[:-1]])
    at, sums = first.copy(), []
    for i in range(per):
        at = at + run[:, i]
        sums.append(at)
    return np.stack(sums, 1), first, cum[31]


@pytest.mark.parametrize("G,threads", [(1, 64), (31, 64), (64, 128), (240, 64), (240, 256), (513, 128)])
def test_sampled_point_against_serial_scan(scan, G, threads):
    rng = np.random.default_rng(G + threads)
    ov = 4.0 / G
    fac = 4.0 / (ov * G)
    grids, us = [], []
    for _ in range(120):
        a = rng.random(G) + 0.1
        b = np.zeros(G)
        off = rng.random(G) < 0.6  # points of probability zero
        off[0::(G + 31) // 32] |= rng.random(len(off[0::(G + 31) // 32])) < 0.7  # and a lane's first point most of the time
        off[rng.integers(G)] = False
        a[off], b[off] = 0.0, 1.0
        grid = np.zeros((G, 4))
        grid[:, 0], grid[:, 1] = a, b
        sums, first, total = lanes(np.where(off, 0.0, a * a) * fac)
        inv = 1.0 / total
        u = [0.0, 1.0 - 2.0**-32, rng.random()]
        gaps = (sums[:-1, -1] * inv)[sums[:-1, -1] < first[1:]]
        u += list(gaps[gaps * 1.0 < 1.0][:4])
        u += [x for x in rng.choice(sums.ravel() * inv, 2) if x < 1.0]
        grids += [grid] * len(u)
        us += u
    grids, us = np.stack(grids), np.array(us)
    index, factor = scan(grids, us, ov, threads)
    pdf = np.maximum(0.0, grids[:, :, 0]**2 - grids[:, :, 1]**2) * fac
    total = pdf.sum(1)
    np.testing.assert_allclose(factor, total, rtol=G * 2.0**-52)
    rows = np.arange(len(us))
    cum = np.cumsum(pdf, 1) / total[:, None]
    tol = G * 2.0**-52
    assert np.all(pdf[rows, index] > 0.0), np.flatnonzero(pdf[rows, index] == 0.0)
    assert np.all(cum[rows, index] > us - tol)
    assert np.all((index == 0) | (cum[rows, np.maximum(index - 1, 0)] <= us + tol))


@pytest.mark.parametrize("G", [1, 31, 240])
def test_pdf_that_sums_to_zero_takes_the_first_point(scan, G):
    grids = np.zeros((3, G, 4))
    grids[:, :, 1] = 1.0
    index, factor = scan(grids, np.array([0.0, 0.5, 1.0 - 2.0**-32]), 4.0 / G, 64)
    assert np.all(index == 0) and np.all(factor == 0.0)
