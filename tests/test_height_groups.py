"""2D strengths over more than one group of 32 evenly spaced heights, where a node's phases may follow by
recurrence in some groups and not in others (exponents past -600 or 80): heights rising and falling,
across a thick layer, and out of the layer they are counted from. FP64 against the oracle, every height on
its own scale, to 1e-9 as the 1D heights past the recurrence are held; the tensor-core precisions against
it to 1e-5 of the height's largest entry (their 24-bit operands are held to 1e-6 of whole fields)."""
import numpy as np
import pytest

from helpers import krho_grid, lay, m_bi, m_gl, m_vac, uniform_phi

pytestmark = pytest.mark.gpu

W = 2 * np.pi


def _stack(d2, d3, d4):
    return [lay(m_vac, 1.0), lay(m_bi, d2), lay(m_gl, d3), lay(m_vac, d4)]


# (thicknesses of layers 2-4, largest kρ, observation layer, heights, source height, terms)
CASES = [
    ((6.0, 0.5, 1.0), 25.0 * W, 2, np.linspace(0.0, 6.0, 128), 3.0, "direct"),
    ((6.0, 0.5, 1.0), 25.0 * W, 2, np.linspace(6.0, 0.0, 96), 2.1, "direct"),
    ((0.8, 0.5, 0.17), 12.0 * W, 4, np.linspace(3.0, 0.0, 64), 0.3, "all"),
    ((0.8, 0.33, 1.0), 12.0 * W, 3, np.linspace(2.5, 0.01, 33), 0.3, "all"),
    ((0.8, 0.5, 1.0), 10.0 * W, 2, np.linspace(-4.0, 0.3, 96), 0.3, "scattered"),
    ((0.8, 0.5, 1.0), 10.0 * W, 2, np.linspace(-4.0, 0.3, 64), 0.2, "all"),
    ((0.8, 0.5, 1.0), 10.0 * W, 2, np.linspace(0.05, 0.75, 65), 0.3, "all"),
]


@pytest.mark.parametrize("ds,kmax,obs,z,zs,terms", CASES)
def test_2d_height_groups(oracle, ds, kmax, obs, z, zs, terms):
    from yellowthinfilms_b200 import api
    st = _stack(*ds)
    kr, wr = krho_grid(st, W, kmax=kmax, width=2.0)
    ph, wp = uniform_phi(5)
    gc = api.build_cavity_transfer_2d(st, W, 2, kr, wr, ph, wp, obs_layers=[obs])
    oc = oracle.build_cavity_transfer_2d(st, W, 2, kr, wr, ph, wp, obs_layers=[obs])
    x, y = np.array([-0.02, 0.0, 0.03]), np.array([0.0, 0.01])
    Go = oracle.closed_form_G(oc, obs, zs, z, x, y, terms=terms)
    scale = np.abs(Go).max(axis=(0, 1, 3, 4))
    assert np.isfinite(scale).all() and (scale > 0).all()
    for precision, tol in (("fp64", 1e-9), ("int8x3", 1e-5), ("split_bf16", 1e-5)):
        if precision == "split_bf16" and scale.max() > 1e30:
            continue  # its operands are FP32 terms
        G = api.closed_form_G(gc, obs, zs, z, x, y, terms=terms, precision=precision)
        err = np.abs(G - Go).max(axis=(0, 1, 3, 4)) / scale
        assert err.max() < tol, (precision, int(err.argmax()), float(err.max()))
