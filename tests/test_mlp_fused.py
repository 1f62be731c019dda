"""The warm-start network's fused training step at the edges of its tiles
(128 rows, 64 columns, rows of 8 elements) and of its rule (widths that are a
multiple of 8, at most 32 outputs; others take the separate kernels)."""
import numpy as np
import pytest

from gelios_2d_b200 import warmstart as W
from oracle import mlp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,depth,n_out,rows", [(64, 2, 5, 1), (64, 2, 5, 129), (72, 3, 3, 127), (8, 1, 1, 300),
                                                     (136, 2, 32, 513), (64, 2, 33, 200), (20, 2, 5, 130)])
def test_gradients(width, depth, n_out, rows):
    """Against the float64 restatement with the device's bf16 roundings: only
    the order of fp32 sums differs (2e-3 of a tensor's norm, as for the
    network of the other gradient test)."""
    net = W.Mlp(7, 6, width, depth, n_out, 600)
    try:
        p = net.init_params(4)
        rng = np.random.default_rng(rows)
        x = rng.uniform(-1, 1, (rows, 7)).astype(np.float32)
        t = rng.normal(size=(rows, n_out)).astype(np.float32)
        loss, g = net.loss_grad(x, t)
        y = net.predict(x)
    finally:
        net.close()
    lay = O.layout(7, 6, width, depth, n_out)
    lb, gb = O.loss_grad(p.astype(np.float64), x, t, 6, lay, bf16_mode=True)
    assert abs(loss - lb) <= 1e-5 * lb
    assert abs(float(((y.astype(np.float64) - t) ** 2).mean()) - loss) <= 1e-5 * lb
    din, dout, w_off, b_off, _ = lay
    for l in range(len(din)):
        for a, n in ((w_off[l], din[l] * dout[l]), (b_off[l], dout[l])):
            assert np.linalg.norm(g[a:a + n] - gb[a:a + n]) <= 2e-3 * np.linalg.norm(gb[a:a + n])


@pytest.mark.parametrize("width,batch", [(64, 500), (20, 130)])
def test_steps_of_one_call_equal_calls_of_one_step(width, batch):
    """A call of several steps replays a captured step; one-step calls enqueue
    it.  Constant learning rate: the same bits."""
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (3000, 7)).astype(np.float32)
    t = rng.normal(size=(3000, 5)).astype(np.float32)
    out = []
    for calls in ((5,), (1,) * 5, (2, 3)):
        net = W.Mlp(7, 6, width, 2, 5, 512)
        try:
            net.init_params(2)
            net.set_data(x, t)
            h = np.concatenate([net.train(k, batch, 1e-3, 1e-3, 0, 9) for k in calls])
            out.append((h, net.params(), net.predict(x)))  # 3000 rows: several chunks
        finally:
            net.close()
    for o in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0], o))
