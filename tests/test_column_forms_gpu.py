"""The column pass over every height, with the packed DC/Nyquist column in its chained form and the kernel
spectrum in either row length: one step through a context (padded, 16-byte aligned rows) and one through
lenia_step_noalloc (the caller's rows of H/2 + 1 values), each against FP64.

U[0,1] over the whole world puts as much into the packed column as into any other, and the stripe along x at
the Nyquist frequency puts more.  Bound: 1e-5 a step, the parity tests'."""
import ctypes

import numpy as np
import pytest

import auto_gb300 as ag
from auto_gb300 import Sim, _lib
from oracle.oracle import fp64_step

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [32, 48, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096])
def test_packed_column_and_both_khat_layouts(h):
    torch = pytest.importorskip("torch")
    w = 64
    k = ag.Kernel(radius=9.0, beta=[1.0, 0.5], mu=0.3, sigma=0.05)
    world = ag.World(w, h, [k], dt=0.1)
    s = np.random.default_rng(h).random((h, w), dtype=np.float32)
    s[:, 1::2] *= np.float32(0.5)
    want = fp64_step(world, s)[0]
    with Sim(world) as sim:
        sim.write_state(0, s)
        sim.step(1)
        assert np.abs(sim.read_state(0)[0] - want).max() < 1e-5
    L = _lib.load()
    khat = np.zeros((w // 2 + 1) * (h // 2 + 1), np.float32)
    kd = world.to_desc().kernels[0]
    assert L.lenia_kernel_spectrum(ctypes.byref(kd), w, h, _lib.fptr(khat), khat.size) == 0
    d_state, d_khat = torch.from_numpy(s.copy()).cuda(), torch.from_numpy(khat).cuda()
    torch.cuda.synchronize()
    assert L.lenia_step_noalloc(ctypes.c_void_p(d_state.data_ptr()), w, h, ctypes.c_void_p(d_khat.data_ptr()), k.mu,
                                k.sigma, world.dt, 1, None) == 0
    torch.cuda.synchronize()
    assert np.abs(d_state.cpu().numpy() - want).max() < 1e-5
