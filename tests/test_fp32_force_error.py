"""The FP32 force's rounding error (relative rms against the FP64 context's force, which the oracle
bounds to 1e-11) is no larger than that of the one-thread-per-link kernels with matrix derivatives
that all FP32 forces took before the plaquette form.  The bars are those kernels' errors on the same
links, as measured with them."""
import numpy as np
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu

DIMS = (8, 8, 8, 8)
# 1e-7 of the force, by links, action and 0 .. 3 stout levels (rho = 0.1)
BARS = {
    ("hot", "iwasaki"): (1.312, 1.631, 2.085, 2.552),
    ("hot", "wilson"): (1.207, 1.539, 1.975, 2.420),
    ("smooth", "iwasaki"): (0.955, 6.897, 26.00, 69.04),
    ("smooth", "wilson"): (0.812, 5.934, 19.14, 44.14),
}


def rough_links(kind):
    """Haar links, or links about 0.3 from the unit matrix (unitary parts of 1 + 0.3 Z, det 1)."""
    U = O.gen_hot(DIMS, 21)
    if kind == "hot":
        return U
    w, _, v = np.linalg.svd(np.eye(3) + 0.3 * U)
    U = w @ v
    return U / np.linalg.det(U)[..., None, None] ** (1.0 / 3.0)


def error(kind, action, n_stout):
    U = rough_links(kind)
    F = []
    for precision in ("fp64", "mixed"):
        with M.Chmc(DIMS, action=action, mag=0, n_stout=n_stout, rho=0.1, precision=precision) as c:
            c.set_gauge(U)
            F.append(c.get_force())
    return np.linalg.norm(F[1] - F[0]) / np.linalg.norm(F[0])


@pytest.mark.parametrize("n_stout", [0, 1, 2, 3])
@pytest.mark.parametrize("kind,action", list(BARS))
def test_fp32_force_is_as_exact_as_the_link_kernels(kind, action, n_stout):
    assert error(kind, action, n_stout) < 1e-7 * BARS[kind, action][n_stout]
