"""Plaquette and rectangle sums at the sizes where the reduction changes shape: a warp per plane
below 49152 (plaquettes alone) and 98304 sites (with rectangles), a thread per site above; for
matrices that are not unitary too.

Bar: 1e-12 relative, the action parity of test_gpu_parity.py (the sums are double-double over
sites; a site's loops round at 1e-15).
"""
import numpy as np
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (3, 5, 3, 3), (8, 12, 16, 31), (8, 12, 16, 32), (8, 16, 24, 31),
                                  (8, 16, 24, 32)])
def test_sums_against_the_oracle(dims):
    U = O.gen_hot(dims, 31)
    U[1, 2] *= 1.5
    p0, r0, _ = O.action(O.make_params(dims, action=1), U)
    with M.Chmc(dims, mag=0, action="iwasaki") as c:
        c.set_gauge(U)
        p, r, _ = c.gauge_action()
        avg = c.avg_plaquette()
    assert abs(p - p0) <= 1e-12 * abs(p0) + 1e-12 and abs(r - r0) <= 1e-12 * abs(r0) + 1e-12
    assert abs(avg - O.avg_plaquette(dims, U)) <= 1e-12 * abs(avg) + 1e-14


def test_a_chain_sums_alike_alone_and_in_an_ensemble():
    """The shape follows the launch's sites; the sums are the same bits."""
    dims = (8, 16, 24, 31)
    with M.Chmc(chains=[dict(dims=dims), dict(dims=(8, 8, 8, 8))], mag=0, seed=4) as e, \
            M.Chmc(dims, mag=0, seed=4) as s:
        for c in (e, s):
            c.hot_start(6)
            c.init_momentum(traj=0)
        assert e.get_hamiltonian(0) == s.get_hamiltonian()
