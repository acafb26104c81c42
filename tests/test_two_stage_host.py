"""The two-stage transforms (auto_gb300/csrc/fft_core.cuh), built for the host with g++, against numpy's FFT.

Bound: relative L2 error 4e-7 on zero-mean data.  A transform of up to 2^8.6 points adds about nine levels of
half-ulp roundings (6e-8 each, independent: 1.8e-7), and its one inter-stage twiddle, a product of at
most four table factors, up to 1e-7 more."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def fft_two(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    out = str(tmp_path_factory.mktemp("fft2") / "fft_two.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC",
                           os.path.join(ROOT, "tests", "cpp", "fft_two_stage_host.cpp"), "-o", out])
    return ctypes.CDLL(out)


@pytest.mark.parametrize("n", [192, 384])
@pytest.mark.parametrize("swapped", [0, 1])
@pytest.mark.parametrize("inverse", [0, 1])
def test_two_stage_matches_numpy(fft_two, n, swapped, inverse):
    rng = np.random.default_rng(n + 2 * swapped + inverse)
    x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    out = np.zeros(n, np.complex64)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert fft_two.fft_two(n, swapped, inverse, ptr(x), ptr(out)) == 0
    x64 = x.astype(np.complex128)
    want = np.fft.ifft(x64) * n if inverse else np.fft.fft(x64)
    assert np.linalg.norm(out - want) / np.linalg.norm(want) < 4e-7
