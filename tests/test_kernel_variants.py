"""Kernel variants chosen where they act on something else than a single context's forces."""
import numpy as np
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [1, 2])
def test_fp64_smearing_variant_reaches_a_mixed_contexts_hamiltonian(levels):
    """The Hamiltonian of a mixed context is smeared in FP64: one launch per level in the chosen
    one-thread-per-link form instead of two, twice per trajectory.  Bar: 1e-12 of the action, its
    parity bar."""
    dims = (4, 4, 4, 6)
    with M.Chmc(dims, mag=2, n_stout=levels, precision="mixed") as c:
        c.set_gauge(O.gen_hot(dims, 8))
        n, s = c.graph_kernel_count(), c.gauge_action()[2]
        c.set_kernel_variant("stout_forward", "fp64", "t1m3")
        assert c.graph_kernel_count() == n - 2 * levels
        assert abs(c.gauge_action()[2] - s) <= 1e-12 * abs(s)
