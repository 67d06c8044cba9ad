"""Small observation sets of a plan at the edges of the batched synthesis kernel: sub-batches of 32 nodes
with a remainder, register tiles of 4 rows x 3 or 1 columns, the node groups (4, 2 or 1 by the number of
tiles), the largest sets, uneven z rows. Against the per-item FP64 synthesis at the plan tests' 1e-12."""
import numpy as np
import pytest

from helpers import FOUNDATION_STACKS, config1_like_stack, relerr

pytestmark = pytest.mark.gpu

W = 2 * np.pi


def _nodes(n, kmax):
    k = kmax * (np.arange(n) + 0.5) / n
    return k, np.full(n, kmax / n)


def _z(nz, even=True):
    return np.linspace(0.02, 0.31, nz) if even else np.sort(np.random.default_rng(nz).uniform(0.02, 0.31, nz))


# (nodes, radii, z rows); the third stack kind: gyrotropic without the symmetry check (13 columns per row)
@pytest.mark.parametrize("n,nr,nz", [(1, 1, 1), (31, 5, 3), (33, 32, 5), (97, 7, 8), (200, 22, 8)])
@pytest.mark.parametrize("kind", ["film", "general"])
@pytest.mark.parametrize("even", [True, False])
def test_1d_sets(n, nr, nz, kind, even):
    from yellowthinfilms_b200 import api
    st = config1_like_stack() if kind == "film" else FOUNDATION_STACKS[4][1]
    k, w = _nodes(n, 6 * W)
    tr = [dict(stack=st, omega=W, source_layer=1, kx_nodes=k, wt_nodes=w, obs_layers=[1, 2], check_symmetry=False)] * 3
    x = np.geomspace(0.01, 2.0, nr)
    ys = [dict(obs_layer=1, zsrc_local=0.03, z_obs=_z(nz, even), xs=x, ys=[0.0]),
          dict(obs_layer=2, zsrc_local=0.03, z_obs=_z(nz, even), xs=x, ys=[0.0]),
          dict(obs_layer=1, zsrc_local=0.1, z_obs=_z(nz, even), xs=x, ys=[0.0], terms="scattered")]
    G = api.BatchPlan(tr, ys)()
    c = api.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1, 2], check_symmetry=False)
    for g, y in zip(G, ys):
        ref = api.closed_form_G(c, y["obs_layer"], y["zsrc_local"], y["z_obs"], y["xs"], y["ys"],
                                terms=y.get("terms", "all"))
        assert relerr(g, ref) < 1e-12


@pytest.mark.parametrize("nk,nphi,nx,ny,nz", [(1, 1, 1, 1, 1), (5, 7, 3, 3, 8), (11, 3, 8, 8, 4), (8, 8, 5, 7, 7),
                                              (9, 11, 2, 16, 2)])
@pytest.mark.parametrize("even", [True, False])
def test_2d_sets(nk, nphi, nx, ny, nz, even):
    from yellowthinfilms_b200 import api
    st = FOUNDATION_STACKS[3][1]
    k, w = _nodes(nk, 6 * W)
    ph, wp = 2 * np.pi * np.arange(nphi) / nphi, np.full(nphi, 2 * np.pi / nphi)
    tr = [dict(stack=st, omega=W, source_layer=2, kr_nodes=k, kr_weights=w, phi_nodes=ph, phi_weights=wp,
               obs_layers=[2, 3])] * 2
    x, y = np.linspace(-0.4, 0.5, nx), np.linspace(-0.3, 0.2, ny)
    ys = [dict(obs_layer=o, zsrc_local=0.1, z_obs=_z(nz, even), xs=x, ys=y) for o in (2, 3)]
    G = api.BatchPlan(tr, ys)()
    c = api.build_cavity_transfer_2d(st, W, 2, k, w, ph, wp, obs_layers=[2, 3], rotation=False)
    for g, it in zip(G, ys):
        ref = api.closed_form_G(c, it["obs_layer"], 0.1, it["z_obs"], x, y)
        assert relerr(g, ref) < 1e-12
