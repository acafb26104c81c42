"""The general row pass (several channels or kernels) in its 80- and its 128-register build: the default (80 where a launch
has between two and three items an SM), equal bits, and a step within 1e-5 of FP64, the parity tests' bound."""
import numpy as np
import pytest

import auto_gb300 as ag
from auto_gb300 import Sim
from oracle.oracle import fp64_step

pytestmark = pytest.mark.gpu


def world(w, h, channels):
    r = 8.0 if min(w, h) >= 64 else 4.0
    kernels = [ag.Kernel(radius=r + 3 * s + d, beta=[1.0, 0.5][: 1 + (s + d) % 2], mu=0.3, sigma=0.06, src=s, dst=d,
                         weight=1.0 / channels)
               for s in range(channels) for d in range(channels)]
    if channels == 1:
        kernels.append(ag.Kernel(radius=r + 7.0, mu=0.25, sigma=0.05, weight=0.5))
    return ag.World(w, h, kernels, channels=channels, dt=0.05)


@pytest.mark.parametrize("w, h, channels, default", [
    (768, 1024, 3, 0),   # 384 items
    (1024, 1024, 3, 0),
    (1536, 1536, 1, 0),
    (768, 768, 3, 1),    # 288
    (1024, 768, 3, 1),
    (512, 1024, 3, 1),   # 384, but six CTAs of 128 threads fit an SM
    (2048, 768, 1, 1),
    # two kernels a target at narrow widths: both inverse transforms at once in the 128-register build, one after
    # the other through the plane in the other
    (32, 64, 1, 1),
    (48, 32, 2, 1),
    (64, 64, 1, 1),
    (96, 128, 2, 1),
    (128, 96, 1, 1),
    (128, 1024, 2, 1),
    (192, 64, 1, 1),
])
def test_general_row_builds(w, h, channels, default):
    wd = world(w, h, channels)
    s = np.random.default_rng(w + h).random((channels, h, w), dtype=np.float32)
    want = np.asarray(fp64_step(wd, s))
    got = []
    for variant in (None, 0, 1):
        with Sim(wd) as sim:
            if variant is None:
                assert [x["row_variant"] for x in sim.shapes().values()] == [default]
            else:
                sim.set_variants(-1, variant)
            sim.write_state(0, s)
            sim.step(1)
            one = sim.read_state(0)
            sim.step(9)
            got.append((one, sim.read_state(0)))
    for one, ten in got:
        assert np.abs(one - want).max() < 1e-5
        np.testing.assert_array_equal(one, got[0][0])
        np.testing.assert_array_equal(ten, got[0][1])
