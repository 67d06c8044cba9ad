"""FP64 2D synthesis whose phase tables (16 (nx + ny) bytes per node) pass their bound of 1 GiB: the nodes go in
passes. Sums in another order than one pass over the pixels in parts: the parity tests' 1e-10 against the
oracle at some pixels, 1e-12 against the parts; and the call's device memory stays bounded."""
import numpy as np
import pytest

from helpers import FOUNDATION_STACKS, relerr, uniform_phi

pytestmark = pytest.mark.gpu

W = 2 * np.pi


def _cache(lib, nk, nphi):
    k = 3 * W * (np.arange(nk) + 0.5) / nk
    ph, wp = uniform_phi(nphi)
    return lib.build_cavity_transfer_2d(FOUNDATION_STACKS[3][1], W, 2, k, np.full(nk, 3 * W / nk), ph, wp, obs_layers=[2])


# 4101 coordinates: passes of 16360 nodes, the last one of 16360, 8 and 1; a column of pixels; more
# coordinates than one pass of 64 nodes
@pytest.mark.parametrize("nk,nphi,nx,ny", [(16360, 2, 4100, 1), (16368, 1, 4100, 1), (5787, 3, 1, 6000),
                                           (16361, 1, 4100, 1), (150, 1, 1200000, 1)])
def test_passes(oracle, nk, nphi, nx, ny):
    from yellowthinfilms_b200 import api
    c = _cache(api, nk, nphi)
    x, y = np.linspace(-0.4, 0.5, nx), np.linspace(-0.3, 0.2, ny)
    z = np.array([0.5])
    G = api.closed_form_G(c, 2, 0.4, z, x, y)
    px, py = np.unique(np.linspace(0, nx - 1, 5).astype(int)), np.unique(np.linspace(0, ny - 1, 5).astype(int))
    oc = _cache(oracle, nk, nphi)
    assert relerr(G[np.ix_(px, py)], oracle.closed_form_G(oc, 2, 0.4, z, x[px], y[py])) < 1e-10
    parts = [api.closed_form_G(c, 2, 0.4, z, x[i:i + 1000], y[j:j + 1000])
             for i in range(0, min(nx, 5000), 1000) for j in range(0, ny, 1000)]
    parts = np.concatenate(parts, axis=0 if nx > 1 else 1)
    assert relerr(G[:parts.shape[0]], parts) < 1e-12


def test_device_memory_is_bounded():
    """65536 nodes x 8192 coordinates: 8 GiB of phase tables in one pass."""
    import torch
    from yellowthinfilms_b200 import api
    ctx = api.Context(0)
    k = 3 * W * (np.arange(65536) + 0.5) / 65536
    ph, wp = uniform_phi(1)
    c = api.build_cavity_transfer_2d(api.Stack(FOUNDATION_STACKS[3][1], ctx), W, 2, k, np.full(65536, 1.0), ph, wp,
                                     obs_layers=[2])
    out = torch.empty(8191 * 9, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    api.closed_form_G(c, 2, 0.4, [0.5], np.linspace(-0.4, 0.5, 8191), [0.0], out=out)
    used = free - torch.cuda.mem_get_info()[0]
    # the tables' 1 GiB, partial sums of at most 444 column and pixel tiles (64 x 9 x 16 bytes), strengths
    assert used < (1 << 30) + 444 * 2 * 64 * 9 * 16 + 65536 * 9 * 16 + 65536 * 12 * 16 + (64 << 20)
    assert torch.isfinite(torch.view_as_real(out)).all().item() and out.abs().max().item() > 0
