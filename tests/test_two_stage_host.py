"""The two-stage transforms and the plans with a merged middle stage (auto_gb300/csrc/fft_core.cuh), built for
the host with g++, against numpy's FFT.

Bound: relative L2 error 4e-7 on zero-mean data.  A transform of up to 2^12.6 points adds about thirteen levels of
half-ulp roundings (6e-8 each, independent: 2.2e-7), and each of its one or two inter-stage twiddles, a
product of at most four table factors, up to 1e-7 more (independent of the other: 1.4e-7)."""
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


def test_merged_plans(fft_two):
    out = (ctypes.c_int * 14)()
    for n, want in ((96, [4, 6, 4]), (384, [8, 6, 8]), (768, [16, 3, 16]), (1536, [16, 6, 16]),
                    (3072, [16, 12, 16]), (6144, [16, 24, 16]), (4096, [16, 16, 16]), (48, [4, 3, 4])):
        k = fft_two.merged_plan(n, out)
        assert list(out[:k]) == want, (n, list(out[:k]))


@pytest.mark.parametrize("n", [96, 384, 1536, 3072, 6144])
@pytest.mark.parametrize("paired", [0, 1])
@pytest.mark.parametrize("inverse", [0, 1])
def test_merged_plan_matches_numpy(fft_two, n, paired, inverse):
    rng = np.random.default_rng(n + 2 * paired + inverse)
    x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    out = np.zeros(n, np.complex64)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    assert fft_two.fft_merged(n, paired, inverse, ptr(x), ptr(out)) == 0
    x64 = x.astype(np.complex128)
    want = np.fft.ifft(x64) * n if inverse else np.fft.fft(x64)
    assert np.linalg.norm(out - want) / np.linalg.norm(want) < 4e-7
