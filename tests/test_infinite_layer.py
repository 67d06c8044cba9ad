"""1D synthesis in a last layer of infinite thickness: its backward wave, counted from z - d, has amplitude 0
and no finite phase. Against the oracle at the synthesis tests' bounds."""
import numpy as np
import pytest

from helpers import config1_like_stack, lay, relerr

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
