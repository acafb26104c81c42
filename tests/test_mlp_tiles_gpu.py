"""The proposer's tile kernel at the edges of its tiles and halves, against the FP64 oracle.

The oracle applies the same bf16 roundings, so what is left is FP32 against FP64 accumulation and the
bf16 values it tips over: a gradient is within 1e-2 of the oracle's in relative L2 norm per tensor, the loss
within 1e-4, a probability within 2e-3 (a tipped bf16 activation moves a logit by 2^-9 of one of its 256
terms)."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu

SLICES = ((M.P_W1, M.P_B1), (M.P_B1, M.P_W2), (M.P_W2, M.P_B2), (M.P_B2, M.P_W3), (M.P_W3, M.P_B3),
          (M.P_B3, M.NPARAM))


@pytest.fixture(scope="module")
def proposer():
    from auto_gb300 import native
    from auto_gb300.screen import Proposer
    native.build()
    p = Proposer(seed=5, max_batch=19585)
    w = p.params()
    rng = np.random.default_rng(2)
    for a, b in ((M.P_B1, M.P_W2), (M.P_B2, M.P_W3), (M.P_B3, M.NPARAM)):
        w[a:b] = 0.05 * rng.standard_normal(b - a)
    p.set_params(w)
    yield p
    p.close()


# one row, a full tile and its neighbours, and one tile more than a CTA per SM takes at once (152 x 128 rows)
@pytest.mark.parametrize("batch", [1, 127, 128, 129, 19585])
def test_gradients_at_tile_edges(proposer, batch):
    rng = np.random.default_rng(batch)
    x = rng.random((batch, M.IN)).astype(np.float32)
    y = (rng.random((batch, M.OUT)) < 0.3).astype(np.float32)
    loss, g = proposer.gradients(x, y)
    want_loss, want = M.loss_and_grads(proposer.params(), x, y)
    assert abs(loss - want_loss) <= 1e-4 * abs(want_loss)
    for a, b in SLICES:
        err = np.linalg.norm(g[a:b] - want[a:b]) / max(np.linalg.norm(want[a:b]), 1e-30)
        assert err < 1e-2, (a, b, err)


# no rows, partial and full tiles, the second tile of a CTA's pipeline, and the edges of the two halves that
# overlap (38912 rows each: two tiles for each of 152 SMs)
@pytest.mark.parametrize("count", [0, 1, 128, 129, 19457, 38912, 38913, 77825])
def test_predict_at_half_edges(proposer, count):
    x = np.random.default_rng(count).random((count, M.IN)).astype(np.float32)
    got = proposer.predict(x)
    assert got.shape == (count, M.OUT)
    if count:
        assert np.abs(got - M.predict(proposer.params(), x)).max() < 2e-3
