"""2D lateral sums at the edges of their tiles (64 and 128 pixels, 8-node stages, column tiles of up to
48 complex columns, node slices of 64 and up) against the FP64 oracle: FP64 to 1e-10, int8x3 to 1e-6
relative, as the parity tests hold them."""
import numpy as np
import pytest

from helpers import FOUNDATION_STACKS, krho_grid, relerr, uniform_phi

pytestmark = pytest.mark.gpu

W = 2 * np.pi


@pytest.mark.parametrize("nk,nphi,nx,ny,nz,even", [(1, 1, 1, 1, 1, True), (7, 1, 3, 1, 2, True), (3, 3, 9, 7, 1, False),
                                                   (13, 5, 13, 5, 5, True), (65, 3, 8, 8, 11, False),
                                                   (130, 7, 33, 2, 6, True)])
@pytest.mark.parametrize("terms", ["all", "scattered"])
def test_lateral_shapes(oracle, nk, nphi, nx, ny, nz, even, terms):
    from yellowthinfilms_b200 import api
    st = FOUNDATION_STACKS[3][1]
    kr, wr = krho_grid(st, W, kmax=14.0, width=0.5)
    kr, wr = np.tile(kr, 2)[:nk], np.tile(wr, 2)[:nk]
    ph, wp = uniform_phi(nphi)
    rng = np.random.default_rng(nk + nx)
    x = np.linspace(-0.4, 0.5, nx) if even else rng.uniform(-0.4, 0.5, nx)
    y = np.linspace(-0.2, 0.3, ny) if even else rng.uniform(-0.2, 0.3, ny)
    z = np.linspace(0.1, 0.75, nz) if even else rng.uniform(0.05, 0.75, nz)
    gc = api.build_cavity_transfer_2d(st, W, 2, kr, wr, ph, wp, obs_layers=[2, 3])
    oc = oracle.build_cavity_transfer_2d(st, W, 2, kr, wr, ph, wp, obs_layers=[2, 3])
    Go = oracle.closed_form_G(oc, 2, 0.4, z, x, y, terms=terms)
    assert relerr(api.closed_form_G(gc, 2, 0.4, z, x, y, terms=terms), Go) < 1e-10
    assert relerr(api.closed_form_G(gc, 2, 0.4, z, x, y, terms=terms, precision="int8x3"), Go) < 1e-6
    if terms == "all":
        G3 = oracle.closed_form_G(oc, 3, 0.4, z / 2, x, y)
        assert relerr(api.closed_form_G(gc, 3, 0.4, z / 2, x, y), G3) < 1e-10
