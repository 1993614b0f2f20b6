"""The proposal network's two-kernel form at the edges of its tiles: one row,
rows around a CTA's 32, sizes that are no multiple of the MMA tiles, against
the FP64 oracle with BF16 emulation (the tolerances of
tests/test_gpu_mcmc.py)."""
import numpy as np
import pytest

from oracle import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nin,H,K,D,batch", [(3, 5, 1, 1, 1), (44, 256, 4, 11, 1), (44, 256, 4, 11, 33),
                                             (7, 40, 3, 2, 64), (30, 31, 8, 5, 100), (16, 64, 2, 3, 257)])
def test_mlp_forms(nin, H, K, D, batch):
    from messi_gb300 import api
    rng = np.random.default_rng(nin * H + batch)
    net = api.MLP(nin, H, K, D, seed=3)
    net.set_params(net.get_params() + rng.normal(0, 0.02, net.nparams).astype(np.float32))
    p = net.get_params().astype(np.float64)
    x, t = rng.normal(size=(batch, nin)), rng.normal(size=(batch, D))
    y = net.forward(x)
    np.testing.assert_allclose(y, mlp_ref.forward(p, x, nin, H, K + 2 * K * D, bf16=True)["y"], rtol=1e-3, atol=1e-4)
    loss, g = net.gradients(x, t)
    loss_ref, g_ref = mlp_ref.gradients(p, x, t, nin, H, K, D, bf16=True)
    assert abs(loss - loss_ref) <= 1e-4 * abs(loss_ref)
    assert np.linalg.norm(g - g_ref) <= 1e-3 * np.linalg.norm(g_ref)
    # a training step moves the packed weights with the master copy
    net.train_step(x, t, lr=1e-2)
    p = net.get_params().astype(np.float64)
    np.testing.assert_allclose(net.forward(x), mlp_ref.forward(p, x, nin, H, K + 2 * K * D, bf16=True)["y"], rtol=1e-3,
                               atol=1e-4)
