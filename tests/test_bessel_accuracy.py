"""Accuracy of the device Bessel functions relative to the value itself, where an absolute bound does not see it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slope", [0.0, 0.2, -0.4, 1.5])
def test_small_arguments(slope):
    """J_n ~ (z/2)^n / n! down to |z| = 1e-9, real and complex: ten roundings and the reference's own error,
    1e-14 relative."""
    from scipy.special import jv
    from yellowthinfilms_b200 import api
    x = np.concatenate([np.geomspace(1e-9, 0.999, 200), [0.25, 0.5, 0.75]])
    z = x * (1 + 1j * slope) / np.hypot(1, slope)
    for n in (0, 1, 2):
        ref = jv(n, z)
        assert (np.abs(api.bessel_j(n, z) - ref) <= 1e-14 * np.abs(ref)).all(), n
    for s in (1, -1):
        j0, j1 = api.bessel_j01(s * x)
        assert (np.abs(j0 - jv(0, x)) <= 1e-14).all()
        assert (np.abs(j1 - s * jv(1, x)) <= 1e-14 * np.abs(jv(1, x))).all()


@pytest.mark.parametrize("lo,hi", [(100.0, 1e3), (1e3, 1e5), (1e5, 8e5)])
def test_real_phase_reduction(lo, hi):
    """J_0, J_1 of large real arguments against Hankel's expansion in extended precision: from x = 100 on the
    five terms taken leave out less than 1e-17, so what is left is rounding, about ten units of 2^-53 of
    the amplitude √(2 / (π x)); the phase's reduction adds at most 2 n 2^-87 (its constant's last part), below
    that on these arguments."""
    from yellowthinfilms_b200 import api
    x = np.concatenate([np.linspace(lo, hi, 4001), np.geomspace(lo, hi, 2000)])
    L = np.longdouble
    xl = x.astype(L)
    pi = L(3) + L("0.14159265358979323846264338327950288")
    ref = []
    for n in (0, 1):
        mu, a, p, q = L(4 * n * n), L(1), L(0), L(0)
        p = p + np.zeros_like(xl)
        q = q + np.zeros_like(xl)
        t = np.ones_like(xl)
        for k in range(14):
            if k:
                t = t * (mu - (2 * k - 1) ** 2) / (8 * k * xl)
            if k % 2 == 0:
                p += t if k % 4 == 0 else -t
            else:
                q += t if k % 4 == 1 else -t
        # χ = x - (2n + 1) π/4 through cos x and sin x, whose reduction is the library's
        c, s = np.cos(xl), np.sin(xl)
        c0, s0 = (c + s) / np.sqrt(L(2)), (s - c) / np.sqrt(L(2))
        cn, sn = (c0, s0) if n == 0 else (s0, -c0)
        ref.append(np.sqrt(2 / (pi * xl)) * (p * cn - q * sn))
    amp = np.sqrt(2 / (np.pi * x))
    for got, r in zip(api.bessel_j01(x), ref):
        err = np.abs(got - r) / amp
        assert err.max() <= 12 * 2.0**-53, float(err.max())
