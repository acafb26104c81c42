"""States in and out through lenia_write_state / lenia_read_state from memory of every kind a caller has: aligned,
4 bytes off, read-only, page-locked and fresh, on both sides of the sizes that the copies are chosen by (64 KiB and 1 MiB).
Copies: equal bits."""
import ctypes
import mmap

import numpy as np
import pytest

import auto_gb300 as ag
from auto_gb300 import Sim
from auto_gb300._lib import fptr

pytestmark = pytest.mark.gpu

SIZES = [(32, 32), (128, 128), (192, 96), (256, 128), (256, 256), (512, 512), (768, 512), (1024, 512)]


def memory(kind, n):
    if kind == "aligned":
        return np.empty(n + 16, np.float32)[:n]
    if kind == "off":
        a = np.empty(n + 16, np.float32)
        k = 1 + (-(a.ctypes.data // 4)) % 4  # 4 bytes past a 16-byte boundary
        assert a[k:].ctypes.data % 16 == 4
        return a[k:k + n]
    if kind == "fresh":  # pages that nobody has touched
        return np.frombuffer(mmap.mmap(-1, 4 * n), np.float32)
    torch = pytest.importorskip("torch")
    return torch.empty(n, pin_memory=True).numpy()


@pytest.mark.parametrize("kind", ["aligned", "off", "fresh", "pinned"])
@pytest.mark.parametrize("w, h", SIZES)
def test_round_trip(w, h, kind):
    n = w * h
    want = np.random.default_rng(n).random(n, dtype=np.float32)
    src, dst = memory(kind, n), memory(kind, n)
    src[:] = want
    src.flags.writeable = False
    with Sim(ag.World(w, h, [ag.Kernel(radius=5.0, mu=0.3, sigma=0.05)], dt=0.1)) as sim:
        step = []
        for _ in range(2):  # the second write follows a step that is still running
            sim._check(sim._L.lenia_write_state(sim._ctx, 0, ctypes.cast(src.ctypes.data, ctypes.POINTER(ctypes.c_float)), n))
            sim._check(sim._L.lenia_read_state(sim._ctx, 0, fptr(dst), n))
            np.testing.assert_array_equal(dst, want)
            sim.step(3)
            step.append(sim.read_state(0))
            sim.step(20)
        np.testing.assert_array_equal(step[0], step[1])
