"""World statistics over sides that divide the CTA's 1024 threads and sides that do not, worlds smaller than one
round of loads and the longest axes, in one context and alone, against FP64.

A thread's float sums run over at most n / 1024 cells: relative error n / 1024 * 2^-24 at worst, 3.5e-5 at 589,824
cells; bound 1e-4, and 1e-4 of a side for the centroid (the patch is compact, so the sums it comes from do not
cancel)."""
import numpy as np
import pytest

import auto_gb300 as ag
from auto_gb300 import Sim

pytestmark = pytest.mark.gpu

SIZES = [(32, 32), (48, 32), (96, 64), (192, 96), (384, 768), (1024, 256), (1536, 32), (96, 6144), (32, 8192), (8192, 32),
         (8192, 64)]


def world(w, h):
    return ag.World(w, h, [ag.Kernel(radius=5.0, mu=0.3, sigma=0.05)], dt=0.1)


def state(w, h):
    """A patch of a quarter of each side across the wrap, with zeros in it."""
    r = np.random.default_rng(w + 3 * h)
    a = np.zeros((h, w), np.float32)
    a[: h // 4, : w // 4] = r.random((h // 4, w // 4), dtype=np.float32)
    a[r.random((h, w)) < 0.3] = 0
    return np.roll(a, (-h // 16, -w // 8), (0, 1))


def want(a):
    a = a.astype(np.float64)
    c = []
    for v in (a.sum(0), a.sum(1)):
        ang = 2 * np.pi * np.arange(v.size) / v.size
        c.append(np.arctan2((v * np.sin(ang)).sum(), (v * np.cos(ang)).sum()) / (2 * np.pi) * v.size % v.size)
    return a.sum(), c[0], c[1]


def check(got, w, h):
    m, x, y = want(state(w, h))
    assert abs(got[0] - m) < 1e-4 * m
    for g, e, n in ((got[1], x, w), (got[2], y, h)):
        d = abs(g - e) % n
        assert min(d, n - d) < 1e-4 * n


@pytest.mark.parametrize("w, h", SIZES)
def test_stats_alone(w, h):
    with Sim(world(w, h)) as sim:
        sim.write_state(0, state(w, h))
        check(sim.stats()[0], w, h)


def test_stats_of_mixed_sizes():
    with Sim([world(w, h) for w, h in SIZES]) as sim:
        for i, (w, h) in enumerate(SIZES):
            sim.write_state(i, state(w, h))
        got = sim.stats()
    for g, (w, h) in zip(got, SIZES):
        check(g, w, h)
