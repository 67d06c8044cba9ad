"""The general-modes pass over several (node, layer) pairs per thread: a stack whose every film needs the
4x4 QR (ε_xz coupling), at a node count where a thread takes several pairs with a remainder, against the
same nodes solved in small sets (one pair per thread): bit for bit."""
import numpy as np
import pytest

from helpers import lay, m_gl, m_vac

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [19001, 45007])
def test_general_modes_pass_over_many_pairs(n):
    from yellowthinfilms_b200 import api
    from yellowthinfilms_b200.materials import GyrotropicMaterial
    tilted = GyrotropicMaterial([[2.3 + 0.01j, 0.1, 0.4], [0.1, 2.9 + 0.01j, 0.2], [0.4, 0.2, 3.4 + 0.02j]])
    st = [lay(m_vac, 1.0), lay(tilted, 0.7), lay(tilted, 0.4), lay(m_gl, 0.5), lay(m_vac, 1.0)]
    W = 2 * np.pi
    k = 6 * W * (np.arange(n) + 0.5) / n
    w = np.full(n, 6 * W / n)
    c = api.build_cavity_transfer_1d(st, W, 2, k, w, obs_layers=[2], check_symmetry=False)
    e = c.export()
    for b in (0, n // 2, n - 500):
        s = slice(b, b + 500)
        p = api.build_cavity_transfer_1d(st, W, 2, k[s], w[s], obs_layers=[2], check_symmetry=False).export()
        for key, ax in (("T", 1), ("basis", 1), ("Qf", 0), ("sf", 0)):
            assert np.array_equal(np.take(e[key], range(b, b + 500), ax), p[key]), key
