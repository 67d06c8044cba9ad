"""The network's forward pass on device memory it cannot use in place: outputs over the inputs, another GPU's
memory. The same outputs, bit for bit, as in memory of their own."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(3, 2), (154, 64, 2), (300, 2)])
@pytest.mark.parametrize("where", ["end", "start", "middle"])
def test_outputs_over_the_inputs(sizes, where):
    import torch
    from yellowthinfilms_b200 import api
    from yellowthinfilms_b200._native import lib
    B, n0 = 60000, sizes[0]
    net = api.MLP(sizes, seed=3)
    X = torch.from_numpy(np.random.default_rng(0).normal(0, 1, (B, n0)).astype(np.float32)).cuda()
    ref = net.forward(X).clone()
    at = {"end": B * (n0 - 2), "start": 0, "middle": (B * (n0 - 2)) // 2}[where]
    out = X.view(-1)[at:at + 2 * B]
    rc = lib().ytf_mlp_forward(net.h, B, ctypes.c_void_p(X.data_ptr()), ctypes.c_void_p(out.data_ptr()), 1)
    assert rc == 0
    assert torch.equal(out.view(B, 2), ref)


def test_memory_of_another_gpu():
    """X and out on another GPU than the network's: reached by copies, as before the fused pass."""
    import torch
    from yellowthinfilms_b200 import api
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    net = api.MLP((17, 33, 2), seed=3)
    X = np.random.default_rng(0).normal(0, 1, (500, 17)).astype(np.float32)
    out = net.forward(torch.from_numpy(X).to("cuda:1"))
    assert out.device.index == 1 and np.array_equal(out.cpu().numpy(), net.forward(X))
