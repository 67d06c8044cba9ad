"""Layers of infinite thickness. The last one: its backward wave, counted from z - d, has amplitude 0 and no
finite phase. The first one, unobserved: its thickness does not enter. And heights that are not numbers, whose
phases count as 0. Against the oracle at the parity tests' bounds."""
import numpy as np
import pytest

from helpers import FOUNDATION_STACKS, config1_like_stack, lay, relerr

pytestmark = pytest.mark.gpu

W = 2 * np.pi


def _rule(n, kmax=6 * W):
    k = kmax * (np.arange(n) + 0.5) / n
    return k, np.full(n, kmax / n)


@pytest.mark.parametrize("z", [np.linspace(0.0, 0.5, 20), np.array([0.01, 0.03, 0.2])])
@pytest.mark.parametrize("terms", ["all", "scattered"])
def test_infinite_last_layer(oracle, z, terms):
    from yellowthinfilms_b200 import api
    st = config1_like_stack()
    st[2] = lay(st[2].eps_material, np.inf)
    k, w = _rule(264)
    gc = api.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[3])
    oc = oracle.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[3])
    x = np.geomspace(0.01, 2.0, 9)
    Go = oracle.closed_form_G(oc, 3, 0.03, z, x, [0.0], terms=terms)
    assert np.isfinite(Go).all() and np.abs(Go).max() > 0
    assert relerr(api.closed_form_G(gc, 3, 0.03, z, x, [0.0], terms=terms), Go) < 1e-10
    assert relerr(api.closed_form_G(gc, 3, 0.03, z, x, [0.0], terms=terms, precision="int8x3"), Go) < 1e-6
    G8 = api.closed_form_G_batch([dict(cache=gc, obs_layer=3, zsrc_local=0.03, z_obs=z, xs=x, ys=[0.0], terms=terms)] * 2,
                                 precision="int8x3")
    assert relerr(G8[1], Go) < 1e-6


def _first(d, aniso):
    st = config1_like_stack() if not aniso else list(FOUNDATION_STACKS[4][1])
    st[0] = lay(st[0].eps_material, d)
    return st


@pytest.mark.parametrize("d", [0.0, np.inf])
@pytest.mark.parametrize("aniso", [False, True])
@pytest.mark.parametrize("obs", [[2], [2, 3]])
def test_first_layer_thickness_does_not_enter(oracle, d, aniso, obs):
    """With source and field in other layers the first layer only reflects: any thickness gives the same
    field, caches and response."""
    from yellowthinfilms_b200 import api
    st, ref = _first(d, aniso), _first(1.0, aniso)
    k, w = _rule(72)
    ph, wp = 2 * np.pi * np.arange(3) / 3, np.full(3, 2 * np.pi / 3)
    x, z = np.array([-0.3, 0.0, 0.2]), np.linspace(0.01, 0.08, 3)
    grid = dict(omega=W, source_layer=2, kr_nodes=k, kr_weights=w, phi_nodes=ph, phi_weights=wp, obs_layers=obs)
    syn = dict(zsrc_local=0.03, z_obs=z, xs=x, ys=x[:2])
    oc = oracle.build_cavity_transfer_2d(ref, W, 2, k, w, ph, wp, obs_layers=obs)
    caches = [api.build_cavity_transfer_2d(st, W, 2, k, w, ph, wp, obs_layers=obs, rotation=r) for r in ("auto", False)]
    caches += api.build_cavity_transfer_batch([dict(grid, stack=st, rotation=False)] * 2)
    for o in obs:
        Go = oracle.closed_form_G(oc, o, 0.03, z, x, x[:2])
        for c in caches:
            assert c.valid.all() and c.Tvalid[o].all()
            assert relerr(api.closed_form_G(c, obs_layer=o, **syn), Go) < 1e-10
        G = api.BatchPlan([dict(grid, stack=st)], [dict(syn, obs_layer=o)])()[0]
        assert relerr(G, Go) < 1e-10
    r = api.cavity_response(ref, W, 2, k)
    # the response's singular values are held to 1e-9 of the oracle elsewhere
    assert np.abs(api.cavity_response(st, W, 2, k) - r).max() <= 1e-9 * r.max()
    assert np.abs(api.cavity_response_batch([(st, W, 2, k)])[0] - r).max() <= 1e-9 * r.max()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("at", [0, 1, 16, 20])
@pytest.mark.parametrize("terms", ["all", "scattered"])
def test_a_height_that_is_not_a_number(oracle, bad, at, terms):
    """Its field is 0, and the other heights' are as without it."""
    from yellowthinfilms_b200 import api
    st = config1_like_stack()
    k, w = _rule(72)
    z = np.sort(np.random.default_rng(1).uniform(0.0, 0.3, 21))
    gc = api.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1, 2])
    oc = oracle.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1, 2])
    x = np.geomspace(0.01, 2.0, 5)
    for o in (1, 2):
        ok = np.arange(21) != at
        Go = oracle.closed_form_G(oc, o, 0.03, z[ok], x, [0.0], terms=terms)
        zb = np.where(ok, z, bad)
        item = dict(cache=gc, obs_layer=o, zsrc_local=0.03, z_obs=zb, xs=x, ys=[0.0], terms=terms)
        for G, tol in ((api.closed_form_G(gc, o, 0.03, zb, x, [0.0], terms=terms), 1e-10),
                       (api.closed_form_G(gc, o, 0.03, zb, x, [0.0], terms=terms, precision="int8x3"), 1e-6),
                       (api.closed_form_G_batch([item] * 2, precision="int8x3")[0], 1e-6)):
            assert (G[:, :, at] == 0).all()
            assert relerr(G[:, :, ok], Go) < tol
