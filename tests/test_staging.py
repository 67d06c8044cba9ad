"""Inputs on both sides of the 2 MiB that one call stages in page-locked memory (131008 nodes of a build, 262143 of a
response, pixel maps of 1D sets, long pixel lines): the same caches and fields, bit for bit, as from their parts."""
import numpy as np
import pytest

from helpers import FOUNDATION_STACKS, config1_like_stack, relerr, uniform_phi

pytestmark = pytest.mark.gpu

W = 2 * np.pi


def _same(big, small, at, n):
    a, b = big.export(), small.export()
    for key in a:
        axis = 1 if key in ("T", "basis") else 0
        assert np.array_equal(np.take(a[key], range(at, at + n), axis=axis), b[key]), key
    assert np.array_equal(big.status()[2][at:at + n], small.status()[2])


@pytest.mark.parametrize("n", [131008, 131009, 200001])
@pytest.mark.parametrize("kind", ["1d", "contour", "2d"])
def test_builds(n, kind):
    from yellowthinfilms_b200 import api
    st = config1_like_stack() if kind != "2d" else FOUNDATION_STACKS[3][1]
    k = 6 * W * (np.arange(n) + 0.5) / n
    if kind == "contour":
        k = k - 0.05j * W * np.sin(np.pi * k / (6 * W))
    w = np.full(n, 1.0) * (1 + 0 * k)
    ph, wp = uniform_phi(1)

    def build(a, b):
        ctx = api.Context(0)
        S = api.Stack(st, ctx)
        if kind == "2d":
            return api.build_cavity_transfer_2d(S, W, 2, k[a:b], w[a:b], ph, wp, obs_layers=[2])
        f = api.build_cavity_transfer_1d_contour if kind == "contour" else api.build_cavity_transfer_1d
        return f(S, W, 1, k[a:b], w[a:b], obs_layers=[1])

    big = build(0, n)
    for at in (0, n - 1000):
        _same(big, build(at, at + 1000), at, 1000)


@pytest.mark.parametrize("n", [262143, 262144])
def test_responses(n):
    from yellowthinfilms_b200 import api
    st = config1_like_stack()
    k = 6 * W * (np.arange(n) + 0.5) / n
    r = api.cavity_response(st, W, 1, k, 0.3, ctx=api.Context(0))
    rb = api.cavity_response_batch([(st, W, 1, k), (st, W, 2, k[:5])], phi=0.3, ctx=api.Context(0))
    part = api.cavity_response(st, W, 1, k[n - 3000:], 0.3)
    assert np.array_equal(r[n - 3000:], part) and np.array_equal(rb[0], r)


@pytest.mark.parametrize("nx", [10000, 250000])
@pytest.mark.parametrize("precision", ["fp64", "int8x3"])
def test_pixel_sets(nx, precision):
    from yellowthinfilms_b200 import api
    k = 3 * W * (np.arange(64) + 0.5) / 64
    w = np.full(64, 3 * W / 64)
    x, z = np.linspace(-3.0, 3.0, nx), np.array([0.1])
    c = api.build_cavity_transfer_2d(FOUNDATION_STACKS[3][1], W, 2, k, w, *uniform_phi(2), obs_layers=[2])
    y = np.array([0.0, 0.2])
    G = api.closed_form_G(c, 2, 0.4, z, x, y, precision=precision)
    part = api.closed_form_G(c, 2, 0.4, z, x[-999:], y, precision=precision)
    tol = 1e-12 if precision == "fp64" else 2e-6  # int8x3 steps the phases of even pixels from the line's first
    assert relerr(G[-999:], part) < tol
    # a map of 2.5 nx pixels onto 25000 radii
    x1 = np.tile(np.linspace(0.001, 3.0, 100), nx // 10000)
    y1 = np.linspace(0.0, 1.0, 250)
    c1 = api.build_cavity_transfer_1d(config1_like_stack(), W, 1, k, w, obs_layers=[1])
    G = api.closed_form_G(c1, 1, 0.03, z, x1, y1, precision=precision)
    part = api.closed_form_G(c1, 1, 0.03, z, x1[-9:], y1[-99:], precision=precision)
    assert relerr(G[-9:, -99:], part) < tol
