"""The fused MLP kernels at the edges of their tiles: row counts around one 128-row tile and over
several tiles per CTA, widths that are not multiples of 16 or 4, one layer, 64-column weight
blocks' remainders, and a layer past 256 (the per-layer GEMMs), against the FP64 restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NETS = [(154, 256, 256, 256, 256, 2), (3, 2), (17, 33, 2), (250, 65, 7, 2), (40, 300, 2)]


def _net(sizes, seed):
    from yellowthinfilms_b200 import api
    net = api.MLP(sizes, seed=seed)
    rng = np.random.default_rng(seed)
    net.params = (net.params + rng.normal(0, 0.02, net.nparam)).astype(np.float32)
    return net


def _case(sizes, rows, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(0, 1, (rows, sizes[0])).astype(np.float32)
    T = np.stack([rng.normal(0, 1, rows), rng.uniform(0, 1, rows)], 1).astype(np.float32)
    return X, T


# FP32 operands carry 16 significant bits (two BF16 terms) into sums of at most 300 terms: 1e-4 of
# the largest output, and of the gradient's norm, as the unfused kernels are held to
@pytest.mark.parametrize("sizes", NETS)
@pytest.mark.parametrize("rows", [1, 127, 129, 20000])
def test_fused_forward_matches_oracle(sizes, rows):
    import torch
    import ytf_mlp_ref as R
    net = _net(sizes, 3)
    X, _ = _case(sizes, rows, 4)
    ref = R.forward(net.params.astype(np.float64), net.sizes, X)[1][-1]
    tol = 1e-4 * max(1.0, np.max(np.abs(ref)))
    assert np.max(np.abs(net.forward(X) - ref)) <= tol
    out = net.forward(torch.from_numpy(X).cuda())
    assert np.max(np.abs(out.cpu().numpy() - ref)) <= tol


@pytest.mark.parametrize("sizes", NETS)
@pytest.mark.parametrize("rows", [1, 65, 3000])
def test_fused_gradients_match_oracle(sizes, rows):
    import ytf_mlp_ref as R
    net = _net(sizes, 5)
    X, T = _case(sizes, rows, 6)
    loss, g = net.gradients(X, T)
    lo, go = R.loss_and_grad(net.params.astype(np.float64), net.sizes, X, T)
    assert abs(loss - lo) <= 1e-5 * max(1.0, abs(lo))
    assert np.linalg.norm(g - go) <= 1e-4 * np.linalg.norm(go)
