"""1D synthesis at the edges of its tiles (32- and 128-row, 32- and 64-column FP64 tiles, k slices of
16 and 64 nodes, the four-lane slice sums from 8 slices on) and at ragged pixel sets, against the
FP64 oracle: FP64 to 1e-10 and int8x3 to 1e-6 relative, as the parity tests hold them."""
import numpy as np
import pytest

from helpers import config1_like_stack, relerr

pytestmark = pytest.mark.gpu

W = 2 * np.pi


def _rule(n, kmax=6 * W):
    x, w = np.polynomial.legendre.leggauss(min(n, 8))
    panels = max(1, n // 8)
    e = np.linspace(0.0, kmax, panels + 1)
    h = 0.5 * np.diff(e)
    k = (0.5 * (e[1:] + e[:-1])[:, None] + h[:, None] * x).ravel()
    wt = (h[:, None] * w).ravel()
    return np.append(k, [])[:n], np.append(wt, [])[:n]


def _case(n, nr, nz, even):
    k, w = _rule(n)
    rng = np.random.default_rng(n + nr + nz)
    z = np.linspace(0.02, 0.31, nz) if even else np.sort(rng.uniform(0.02, 0.31, nz))
    return k, w, np.geomspace(0.01, 3.0, nr), z


@pytest.mark.parametrize("n,nr,nz,even", [(1, 1, 1, True), (7, 33, 3, False), (17, 31, 17, True), (65, 129, 2, False),
                                          (264, 8, 4, True), (4104, 251, 61, True), (8200, 129, 33, False)])
@pytest.mark.parametrize("terms", ["all", "scattered"])
def test_1d_synthesis_shapes(oracle, n, nr, nz, even, terms):
    from yellowthinfilms_b200 import api
    st = config1_like_stack()
    k, w, rho, z = _case(n, nr, nz, even)
    gc = api.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1, 2])
    oc = oracle.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1, 2])
    Go = oracle.closed_form_G(oc, 1, 0.03, z, rho, [0.0], terms=terms)
    assert relerr(api.closed_form_G(gc, 1, 0.03, z, rho, [0.0], terms=terms), Go) < 1e-10
    assert relerr(api.closed_form_G(gc, 1, 0.03, z, rho, [0.0], terms=terms, precision="int8x3"), Go) < 1e-6
    if terms == "all":  # another layer's field, a pixel patch off the axis
        x, y = np.linspace(-0.4, 0.5, 5), np.linspace(-0.3, 0.2, 3)
        G2 = oracle.closed_form_G(oc, 2, 0.03, z / 4, x, y)
        assert relerr(api.closed_form_G(gc, 2, 0.03, z / 4, x, y), G2) < 1e-10
        G8 = api.closed_form_G_batch([(gc, 2, 0.03, z / 4, x, y)], precision="int8x3")[0]
        assert relerr(G8, G2) < 1e-6


def test_1d_general_columns_without_the_symmetry_check(oracle):
    """A gyrotropic stack on a 1D rule (check_symmetry=False): every coefficient column in use."""
    from helpers import FOUNDATION_STACKS
    from yellowthinfilms_b200 import api
    st = FOUNDATION_STACKS[4][1]  # gyrotropic: x and y sources couple
    k, w, rho, z = _case(264, 33, 5, True)
    gc = api.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1], check_symmetry=False)
    oc = oracle.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1])
    Go = oracle.closed_form_G(oc, 1, 0.03, z, rho, [0.1], terms="scattered")
    assert np.abs(Go[..., 1, 0]).max() > 1e-6 * np.abs(Go).max()
    assert relerr(api.closed_form_G(gc, 1, 0.03, z, rho, [0.1], terms="scattered"), Go) < 1e-10
    assert relerr(api.closed_form_G(gc, 1, 0.03, z, rho, [0.1], terms="scattered", precision="int8x3"), Go) < 1e-6
    G8 = api.closed_form_G_batch([(gc, 1, 0.03, z, rho, [0.1])] * 2, precision="int8x3")
    assert relerr(G8[1], oracle.closed_form_G(oc, 1, 0.03, z, rho, [0.1])) < 1e-6


@pytest.mark.parametrize("d,z,obs,terms", [(17.0, np.linspace(0.0, 16.9, 9), 1, "direct"),
                                           (17.0, np.geomspace(0.01, 16.9, 7), 1, "direct"),
                                           (0.33, np.linspace(-4.0, 0.07, 20), 2, "all"),
                                           (0.33, np.linspace(-4.0, 0.3, 20), 1, "scattered")])
def test_1d_heights_past_the_phase_recurrence(oracle, d, z, obs, terms):
    """Exponents below -600 (a 17 λ air layer, its direct term: the rows' own exponentials) and above
    80 (heights below the layer: the general columns' clamped phases)."""
    from helpers import lay
    from yellowthinfilms_b200 import api
    from yellowthinfilms_b200.materials import IsotropicMaterial
    st = config1_like_stack()
    st[0] = lay(IsotropicMaterial(1.0), d)
    k, w, rho, _ = _case(264, 9, 3, True)
    gc = api.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1, 2])
    oc = oracle.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1, 2])
    Go = oracle.closed_form_G(oc, obs, 0.03, z, rho, [0.0], terms=terms)
    G = api.closed_form_G(gc, obs, 0.03, z, rho, [0.0], terms=terms)
    assert relerr(G, Go) < 1e-10
    for i in range(len(z)):  # every height on its own scale
        assert relerr(G[:, :, i], Go[:, :, i]) < 1e-9 or np.linalg.norm(Go[:, :, i]) < 1e-280


def test_bessel_pair_of_the_images():
    """J_0, J_1 of the digit images: the Taylor rows to 4 units of 1 (their rounding) below 25, at row
    edges and centres, the asymptotic pair to 1e-12 from 25 on, odd and even for negative x."""
    from scipy.special import j0, j1
    from yellowthinfilms_b200 import api
    e = np.arange(26.0)
    x = np.concatenate([[0.0], np.linspace(0, 25, 5001)[:-1], e[1:] - 1e-14 * e[1:], e[:-1] + 0.5])
    a, b = api.bessel_j01(np.concatenate([x, -x]))
    tol = 4 * 2.3e-16 + 4e-16  # and the reference's own error
    assert np.abs(a - np.tile(j0(x), 2)).max() <= tol
    assert np.abs(b - np.concatenate([j1(x), -j1(x)])).max() <= tol
    x = np.concatenate([np.linspace(25, 60, 3001), np.geomspace(60, 1e5, 3001)])
    a, b = api.bessel_j01(x)
    assert np.abs(a - j0(x)).max() <= 1e-12 and np.abs(b - j1(x)).max() <= 1e-12


@pytest.mark.parametrize("im", [0.0, 1e-3, 0.4, 0.41, 3.0, 30.0])
def test_complex_bessel_ranges(im):
    """J_0, J_1, J_2 of z = x ± i im on both sides of every range: Taylor rows (0 <= x < 25 up to
    |im| = 0.4, row edges at whole x), series (|z| <= 8), recurrence, asymptotic expansion (|z| >= 25).
    The series' largest term is e^8 / √(16π) ≈ 4e2 of 2^-53 each: 1e-13 relative to e^|im| covers it."""
    from scipy.special import jv
    from yellowthinfilms_b200 import api
    x = np.concatenate([np.linspace(0.0, 60.0, 1201), np.arange(1, 27) - 1e-9, [24.9999999, 25.0000001, 180.3]])
    for sign in (1, -1):
        z = x + 1j * sign * im
        for n in (0, 1, 2):
            assert np.abs(api.bessel_j(n, z) - jv(n, z)).max() < 1e-13 * np.exp(im)


@pytest.mark.parametrize("edge", [0.0, 1e-9, 0.5, 1.0, 2.0, 24.0, 25.0, 500.0])
def test_real_bessel_ranges_of_the_fp64_tables(oracle, edge):
    """FP64 1D synthesis with k ρ on both sides of an edge of the J_n ranges (series below 1, Taylor rows
    at whole arguments, Hankel's expansion from 25), at the tolerance of the shapes above."""
    from yellowthinfilms_b200 import api
    st = config1_like_stack()
    k, w = _rule(8)
    gc = api.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1])
    oc = oracle.build_cavity_transfer_1d(st, W, 1, k, w, obs_layers=[1])
    rho = edge / k[3] * np.array([1 - 1e-12, 1.0, 1 + 1e-12])
    Go = oracle.closed_form_G(oc, 1, 0.03, [0.05, 0.1], rho, [0.0])
    assert relerr(api.closed_form_G(gc, 1, 0.03, [0.05, 0.1], rho, [0.0]), Go) < 1e-10


@pytest.mark.parametrize("n", [450, 6001, 11003])
def test_int8_slices_of_every_length(n):
    """The coefficient images' blocks by slice length (up to 512 nodes, 10000, above) with a ragged last
    stage: int8x3 against the FP64 synthesis of the same cache, at the shapes' 1e-6."""
    from yellowthinfilms_b200 import api
    k = 6 * W * (np.arange(n) + 0.5) / n
    c = api.build_cavity_transfer_1d(config1_like_stack(), W, 1, k, np.full(n, 6 * W / n), obs_layers=[1])
    z, x = np.linspace(0.0, 0.3, 256), np.geomspace(0.01, 3.0, 2048)
    G = api.closed_form_G(c, 1, 0.03, z, x, [0.0], terms="scattered", precision="int8x3")
    assert relerr(G, api.closed_form_G(c, 1, 0.03, z, x, [0.0], terms="scattered")) < 1e-6


@pytest.mark.parametrize("panels,nr", [(3, 1), (17, 9), (65, 131)])
def test_int8_contour_shapes(panels, nr):
    """The complex J digit images at ragged rows (row groups of 8 in tiles of 128) and node counts (stages of
    64): int8x3 on the deformed contour against its FP64 synthesis, at the shapes' 1e-6."""
    from yellowthinfilms_b200 import api
    st = config1_like_stack()
    k, w = api.contour_rule(W, npanels=panels)
    c = api.build_cavity_transfer_1d_contour(st, W, 1, k, w, obs_layers=[1])
    x, z = np.geomspace(0.01, 3.0, nr), np.linspace(0.05, 0.3, 5)
    G = api.closed_form_G(c, 1, 0.03, z, x, [0.0], precision="int8x3")
    assert relerr(G, api.closed_form_G(c, 1, 0.03, z, x, [0.0], precision="fp64")) < 1e-6
