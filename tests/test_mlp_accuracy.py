"""Error of the node placement network's gradients against 64 bits, batch by batch size: no more than with one GEMM
per layer and K slice, whose errors on these networks were 3.8e-6, 3.9e-6, 5.8e-6 and 8.0e-6 of the
gradient's norm (rounded up from the measured means)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,tol", [(512, 3.8e-6), (2048, 3.9e-6), (8192, 5.8e-6), (40000, 8.0e-6)])
def test_gradient_error(B, tol):
    import ytf_mlp_ref as R
    from yellowthinfilms_b200 import api
    err = []
    for seed in range(4):
        rng = np.random.default_rng(seed + 100)
        net = api.MLP((154, 256, 256, 256, 256, 2), seed=seed)
        net.params = (net.params + rng.normal(0, 0.02, net.nparam)).astype(np.float32)
        X = rng.normal(0, 1, (B, 154)).astype(np.float32)
        T = np.stack([rng.normal(0, 1, B), rng.uniform(0, 1, B)], 1).astype(np.float32)
        g = net.gradients(X, T)[1]
        ref = R.loss_and_grad(net.params.astype(np.float64), net.sizes, X, T)[1]
        err.append(np.linalg.norm(g - ref) / np.linalg.norm(ref))
    assert np.mean(err) <= tol, np.mean(err)
