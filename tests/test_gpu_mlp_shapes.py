"""Gradients and training of the surrogate's MLP at the edges of its fused kernels: one row,
rows and columns around 8, 32 and 256, narrow and wide outputs, few and many inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(4, 64, 1, 1), (4, 64, 1, 256), (3, 72, 9, 7), (4, 40, 33, 257), (4, 256, 2100, 64),
          (4, 64, 2049, 31), (20, 64, 40, 300), (15, 33, 17, 65)]


@pytest.mark.parametrize("n_in,H,n_out,rows", SHAPES)
def test_gradients(cilib, n_in, H, n_out, rows):
    """Against the FP64 oracle with the BF16 weights: operands of every product are BF16 (2^-8
    per value), the sums FP32: 3e-2 of the gradient and 2e-2 of the loss, as elsewhere."""
    torch = pytest.importorskip("torch")
    import mlp_oracle
    from cppimpact_gb300 import surrogate as sg
    rng = np.random.default_rng(rows + n_out)
    X = rng.uniform(-1, 1, (rows, n_in)).astype(np.float32)
    T = rng.standard_normal((rows, n_out)).astype(np.float32)
    net = sg.MLP(n_in, H, n_out, seed=5)
    pb = torch.tensor(net.params()).to(torch.bfloat16).float().numpy()
    g, loss = net.gradients(torch.tensor(X, device="cuda"), torch.tensor(T, device="cuda"))
    loss_ref, g_ref = mlp_oracle.loss_and_grad(pb, X, T, n_in, H, n_out)
    assert loss == pytest.approx(loss_ref, rel=2e-2)
    o = 0
    for size in (n_in * H, H, H * H, H, H * n_out, n_out):
        a, b = g[o:o + size], g_ref[o:o + size]
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(g_ref)
        o += size


@pytest.mark.parametrize("n_in,H,n_out,rows", SHAPES)
def test_one_step_is_adam_on_the_gradients(cilib, n_in, H, n_out, rows):
    """One full-batch step: parameters after it are Adam's first step on ci_mlp_gradients'
    gradients (the mini-batch shuffles the rows, which reorders FP32 sums: a gradient entry
    near zero may turn, so all but a thousandth of the entries agree to 1e-3 of the step),
    and the BF16 copies that the next prediction reads are the new parameters'."""
    torch = pytest.importorskip("torch")
    from cppimpact_gb300 import surrogate as sg
    rng = np.random.default_rng(7 * rows + n_out)
    X = torch.tensor(rng.uniform(-1, 1, (rows, n_in)).astype(np.float32), device="cuda")
    T = torch.tensor(rng.standard_normal((rows, n_out)).astype(np.float32), device="cuda")
    net = sg.MLP(n_in, H, n_out, seed=9)
    p0 = net.params().astype(np.float64)
    g, _ = net.gradients(X, T)
    g = g.astype(np.float64)
    lr = 1e-3
    net.train(X, T, 1, rows, lr, 1)
    p1 = net.params()
    step = lr * g / (np.abs(g) + 1e-8)
    off = np.abs(p1 - (p0 - step)) > 1e-3 * lr + 2.0 ** -23 * np.abs(p0)
    assert off.mean() <= 1e-3 + 2.0 / off.size
    other = sg.MLP(n_in, H, n_out, seed=10)
    other.set_params(p1)
    assert torch.equal(net.predict(X), other.predict(X))
