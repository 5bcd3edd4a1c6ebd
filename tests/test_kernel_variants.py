"""Kernel variants chosen where they act on something else than a single context's forces."""
import ctypes

import numpy as np
import pytest

import mag_b200 as M
import oracle as O
from mag_b200._lib import check
from mag_b200.dd import DomainChmc

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


@pytest.mark.parametrize("rank", [0, 1])
@pytest.mark.parametrize("n_stout", [0, 2])
def test_one_shard_of_a_split_lattice_in_the_other_form(rank, n_stout):
    """A variant chosen for one shard: it is tuned without the others, and the shards still meet at the
    same exchanges although their forces are of different forms.  Bar: the force parity bar."""
    dims, halo = (4, 4, 4, 8), 2
    U = O.gen_hot(dims, 10)
    with DomainChmc(dims, 2, halo, mag=2, n_stout=n_stout) as d:
        d.set_gauge(U)
        ctx = ctypes.c_void_p()
        check(d._lib.mag_dd_shard(d._h, rank, ctypes.byref(ctx)), "mag_dd_shard")
        check(d._lib.mag_set_kernel_variant(ctx, b"staple", 0, b"t1m3"), "mag_set_kernel_variant")
        F = d.get_force()
    F0 = O.force(O.make_params(dims, mag=2, action=1, n_stout=n_stout, rho=0.1), U)
    assert np.abs(F - F0).max() < 1e-11 * max(1.0, np.abs(F0).max())
