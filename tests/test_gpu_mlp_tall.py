"""Gradients over more rows than one CTA passes over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,H,n_out,rows", [(4, 40, 9, 16384), (4, 40, 9, 16385), (20, 33, 2050, 16400),
                                               (3, 64, 1, 50001)])
def test_gradients(cilib, n_in, H, n_out, rows):
    """Against the FP64 oracle with the BF16 weights, bounds as in tests/test_gpu_mlp_shapes.py,
    and the same bits twice."""
    torch = pytest.importorskip("torch")
    import mlp_oracle
    from cppimpact_gb300 import surrogate as sg
    rng = np.random.default_rng(rows + n_out)
    X = rng.uniform(-1, 1, (rows, n_in)).astype(np.float32)
    T = rng.standard_normal((rows, n_out)).astype(np.float32)
    net = sg.MLP(n_in, H, n_out, seed=5)
    pb = torch.tensor(net.params()).to(torch.bfloat16).float().numpy()
    dX, dT = torch.tensor(X, device="cuda"), torch.tensor(T, device="cuda")
    g, loss = net.gradients(dX, dT)
    again, _ = net.gradients(dX, dT)
    assert np.array_equal(g, again)
    loss_ref, g_ref = mlp_oracle.loss_and_grad(pb, X, T, n_in, H, n_out)
    assert loss == pytest.approx(loss_ref, rel=2e-2)
    o = 0
    for size in (n_in * H, H, H * H, H, H * n_out, n_out):
        a, b = g[o:o + size], g_ref[o:o + size]
        assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(g_ref)
        o += size
    net.close()
