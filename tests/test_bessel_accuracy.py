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
