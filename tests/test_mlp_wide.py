"""GEMMs whose K goes around the ring of stages (more than 256): wide layers,
and weight gradients of batches above 8192 rows."""
import numpy as np
import pytest

from gelios_2d_b200 import _native as N
from gelios_2d_b200 import warmstart as W
from oracle import mlp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [8, 64, 256, 264, 320, 512, 520, 1000, 1024, 4096])
@pytest.mark.parametrize("M,Nn", [(128, 64), (333, 200)])
def test_gemm(M, Nn, K):
    """Rows of a multiple of 8 (the TMA path); the bound of the other GEMM
    test."""
    import torch

    g = torch.Generator().manual_seed(M + Nn + K)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16)
    B = torch.randn(Nn, K, generator=g).to(torch.bfloat16)
    ref = A.double() @ B.double().t()
    Ad, Bd = A.cuda(), B.cuda()
    C = torch.full((M, Nn), float("nan"), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    for _ in range(3):
        N.check(N.lib().gelios_mlp_gemm_bf16(M, Nn, K, Ad.data_ptr(), K, Bd.data_ptr(), K, C.data_ptr(), Nn, None), "gemm")
        err = (C.double().cpu() - ref).abs().max().item()
        assert err <= 1e-5 * ref.abs().max().item() * max(1.0, K / 64), err


@pytest.mark.parametrize("width,depth,n_out,rows", [(264, 2, 5, 300), (512, 3, 1, 1000), (1024, 2, 32, 500),
                                                    (512, 2, 40, 300), (64, 2, 5, 20000), (40, 1, 3, 70000)])
def test_network(width, depth, n_out, rows):
    """Gradients, loss and prediction against the float64 restatement with the
    device's bf16 roundings; the bounds of the narrow networks' test."""
    net = W.Mlp(7, 6, width, depth, n_out, rows)
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


@pytest.mark.parametrize("width,batch", [(512, 700), (64, 20000)])
def test_training(width, batch):
    """Steps of one call are those of one-step calls, and the loss falls."""
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (batch, 7)).astype(np.float32)
    t = np.tanh(x[:, :5] * 2).astype(np.float32)
    out = []
    for calls in ((6,), (1,) * 6):
        net = W.Mlp(7, 6, width, 2, 5, batch)
        try:
            net.init_params(2)
            net.set_data(x, t)
            h = np.concatenate([net.train(k, batch, 1e-3, 1e-3, 0, 9) for k in calls])
            out.append((h, net.params()))
        finally:
            net.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert out[0][0][-1] < out[0][0][0]
