"""The proposer's results in the caller's memory of every kind (aligned, 4 bytes off, page-locked, fresh), on both sides of the
1 MiB up to which kernels write it in place (87,381 rows of three probabilities).

Probabilities: a row's arithmetic does not depend on where it goes: equal bits.  Gradients: tiles meet in float additions of
any order; 8 tiles of sums below 1 differ by at most 8 * 2^-24 of the sums' magnitude; bound 2e-6 of each tensor's largest."""
import ctypes
import mmap

import numpy as np
import pytest

from auto_gb300.screen import Proposer

pytestmark = pytest.mark.gpu
P = ctypes.POINTER(ctypes.c_float)


def memory(kind, n):
    if kind == "aligned":
        return np.full(n + 16, np.nan, np.float32)[:n]
    if kind == "off":
        a = np.full(n + 16, np.nan, np.float32)
        k = 1 + (-(a.ctypes.data // 4)) % 4
        return a[k:k + n]
    if kind == "fresh":
        return np.frombuffer(mmap.mmap(-1, 4 * n), np.float32)
    torch = pytest.importorskip("torch")
    return torch.full((n,), float("nan"), pin_memory=True).numpy()


def ptr(a):
    return ctypes.cast(a.ctypes.data, P)


@pytest.mark.parametrize("rows", [1, 127, 1000, 87381, 87382])
def test_probabilities(rows):
    p = Proposer(seed=3, max_batch=1024)
    x = np.random.default_rng(rows).random((rows, 16), dtype=np.float32)
    got = []
    for kind in ("off", "aligned", "fresh", "pinned"):
        out = memory(kind, 3 * rows)
        assert p.L.lenia_mlp_predict(p.h, ptr(x), rows, ptr(out)) == 0
        got.append(out.copy())
    assert np.isfinite(got[0]).all()
    for g in got[1:]:
        np.testing.assert_array_equal(g, got[0])


@pytest.mark.parametrize("rows", [1, 1000])
def test_gradients(rows):
    p = Proposer(seed=3, max_batch=1024)
    r = np.random.default_rng(rows)
    x, y = r.random((rows, 16), dtype=np.float32), (r.random((rows, 3)) < 0.3).astype(np.float32)
    got = []
    for kind in ("off", "aligned", "fresh", "pinned"):
        out, loss = memory(kind, p.nparam), ctypes.c_float()
        assert p.L.lenia_mlp_gradients(p.h, ptr(x), ptr(y), rows, ptr(out), ctypes.byref(loss)) == 0
        got.append(out.copy())
    for lo, hi in ((0, 4096), (4096, 4352), (4352, 69888), (69888, 70144), (70144, 70912), (70912, 70915)):
        top = np.abs(got[0][lo:hi]).max()
        assert top > 0
        for g in got[1:]:
            assert np.abs(g[lo:hi] - got[0][lo:hi]).max() <= 2e-6 * top


@pytest.mark.parametrize("shift", [1, 2, 4, 8])
def test_rows_and_labels_at_any_address(shift):
    """Inputs `shift` bytes past a 16-byte boundary give what aligned ones give."""
    rows, r = 300, np.random.default_rng(shift)
    x, y = r.random((rows, 16), dtype=np.float32), (r.random((rows, 3)) < 0.3).astype(np.float32)
    p = Proposer(seed=3, max_batch=512)

    def moved(a):
        b = np.zeros(a.nbytes + 64, np.uint8)
        k = -b.ctypes.data % 16 + shift
        b[k:k + a.nbytes] = a.view(np.uint8).reshape(-1)
        return b, ctypes.cast(b.ctypes.data + k, P)

    (bx, px), (by, py) = moved(x), moved(y)
    got = []
    for ax, ay in ((ptr(x), ptr(y)), (px, ptr(y)), (ptr(x), py), (px, py)):
        out, probs, loss = np.empty(p.nparam, np.float32), np.empty(3 * rows, np.float32), ctypes.c_float()
        assert p.L.lenia_mlp_gradients(p.h, ax, ay, rows, ptr(out), ctypes.byref(loss)) == 0
        assert p.L.lenia_mlp_predict(p.h, ax, rows, ptr(probs)) == 0
        got.append((out, probs, loss.value))
    for g, q, l in got[1:]:
        np.testing.assert_array_equal(q, got[0][1])
        assert np.abs(g - got[0][0]).max() <= 2e-6 * np.abs(got[0][0]).max() and abs(l - got[0][2]) <= 1e-6


def test_probabilities_over_their_own_rows():
    rows = 20000
    x = np.random.default_rng(1).random((rows, 16), dtype=np.float32)
    p = Proposer(seed=3, max_batch=512)
    want, buf = np.empty(3 * rows, np.float32), x.reshape(-1).copy()
    assert p.L.lenia_mlp_predict(p.h, ptr(x), rows, ptr(want)) == 0
    assert p.L.lenia_mlp_predict(p.h, ptr(buf), rows, ptr(buf)) == 0
    np.testing.assert_array_equal(buf[:3 * rows], want)


# copied where the rows are not 16-byte aligned, in halves of 38,912 rows that overlap: one, two, three (the first half's
# buffers used again) and four of them, with a short last one
@pytest.mark.parametrize("count", [1, 38912, 38913, 77824, 77825, 116737, 150001])
def test_copied_halves_give_the_bits_of_rows_in_place(count):
    p = Proposer(seed=3, max_batch=64)
    x = np.random.default_rng(count).random((count, 16), dtype=np.float32)
    off = memory("off", 16 * count)
    off[:] = x.reshape(-1)
    got = []
    for rows in (x, off):
        for kind in ("aligned", "pinned"):
            out = memory(kind, 3 * count)
            assert p.L.lenia_mlp_predict(p.h, ptr(rows), count, ptr(out)) == 0
            got.append(out.copy())
    assert np.isfinite(got[0]).all()
    for g in got[1:]:
        np.testing.assert_array_equal(g, got[0])


def test_rows_in_place_in_two_launches():
    """One row more than a launch takes (2^20): the rows of both launches give what they give in a call of their own."""
    count, cut = (1 << 20) + 1, 1 << 19
    p = Proposer(seed=3, max_batch=64)
    x = np.random.default_rng(2).random((count, 16), dtype=np.float32)
    got = p.predict(x)
    np.testing.assert_array_equal(got[:cut], p.predict(x[:cut]))
    np.testing.assert_array_equal(got[cut:], p.predict(x[cut:]))


@pytest.mark.parametrize("count, at", [(20000, 0.5), (150001, 1.0), ((1 << 20) + 1, 1.0)])
def test_probabilities_over_later_rows(count, at):
    """Probabilities from the middle or at the end of their own rows."""
    p = Proposer(seed=3, max_batch=64)
    x = np.random.default_rng(3).random((count, 16), dtype=np.float32)
    want, k = p.predict(x), int(at * 13 * count) // 4 * 4
    for kind in ("aligned", "off"):
        buf = memory(kind, 16 * count)
        buf[:] = x.reshape(-1)
        assert p.L.lenia_mlp_predict(p.h, ptr(buf), count, ptr(buf[k:])) == 0
        np.testing.assert_array_equal(buf[k:k + 3 * count].reshape(-1, 3), want)
