"""Overlapped launches of the step (programmatic dependent launches, in the step graphs or one by one)
against the same passes launched one after another (lenia_profile_step): the arithmetic is the same, so
the states must be equal bit for bit."""
import numpy as np
import pytest

import auto_gb300 as ag
from auto_gb300.program import Kernel, Seed, World

pytestmark = pytest.mark.gpu


def _world(w, h, channels=1):
    r = min(9.0, min(w, h) // 2 - 1)
    kernels = [Kernel(radius=r, mu=0.2, sigma=0.04, src=s, dst=d, weight=1.0 / channels)
               for s in range(channels) for d in range(channels)]
    return World(w, h, kernels, channels=channels, dt=0.05, seed=Seed("patches", [(w // 4, h // 4, w // 2, h // 2)]))


# launches of at most one CTA an SM, in between, and of many small CTAs (the three sides of the rule for
# early dependents), several waves, both plan kinds of the column pass, chunks on lanes, the general step
@pytest.mark.parametrize("worlds", [
    [(32, 32, 1, 1)], [(128, 128, 1, 1)], "smoothlife", [(1024, 1024, 1, 1)], [(1536, 768, 1, 1)],
    [(128, 128, 1, 40)], [(192, 192, 1, 70)], [(4096, 4096, 1, 1)], [(64, 8192, 1, 1)], [(1024, 1024, 1, 12)],
    [(256, 256, 3, 1)], [(1024, 128, 2, 40)], [(128, 128, 1, 5), (512, 512, 1, 3), (96, 384, 1, 2)],
])
def test_overlapped_step_gives_the_bits_of_separate_launches(worlds):
    if worlds == "smoothlife":
        made = [ag.smoothlife(512, 256)]
    else:
        made = [_world(w, h, c) for w, h, c, n in worlds for _ in range(n)]
    got = []
    for overlapped in (True, False):
        with ag.Sim(made, seed=3) as sim:
            for steps in (75, 3):  # a whole graph, eight generations and single ones (or direct launches), then single ones
                sim.step(steps) if overlapped else sim.profile(steps)
            got.append(sim.read_states())
    assert np.array_equal(got[0], got[1])
    assert got[0].max() > 0
