"""The stout derivative on plaquettes (kernels_smear.cu) where it can go wrong: partial tiles,
extents of two, exponents beyond the series (halved first), and exponents that are exactly zero
(Lambda = 0, field-multi.h:190), against the oracle's literal chain rule.

Bars: the force parity bars of test_gpu_parity.py, 1e-11 of the largest force component in FP64
and 5e-5 in mixed precision; halving adds a few roundings to each Lambda, far inside both.
"""
import numpy as np
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu


def _check(dims, U, precision, tol, **kw):
    F0 = O.force(O.make_params(dims, mag=kw["mag"], action=1, n_stout=kw["n_stout"], rho=kw["rho"]), U)
    with M.Chmc(dims, action="iwasaki", precision=precision, **kw) as c:
        c.set_gauge(U)
        F = c.get_force()
    assert np.abs(F - F0).max() < tol * max(1.0, np.abs(F0).max())


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 5e-5)])
@pytest.mark.parametrize("dims,mag,n_stout,rho", [
    ((5, 3, 3, 4), 0, 2, 0.1), ((2, 2, 2, 2), 2, 1, 0.1), ((2, 6, 4, 3), 0, 3, 0.1),
    ((4, 4, 4, 4), 2, 1, 0.8), ((3, 4, 5, 2), 0, 1, 3.0)])
def test_force_on_edges_and_large_exponents(dims, mag, n_stout, rho, precision, tol):
    _check(dims, O.gen_hot(dims, 11), precision, tol, mag=mag, n_stout=n_stout, rho=rho)


def test_zero_exponents_give_zero_lambda():
    """One rough link in a unit lattice: most exponents are exactly zero."""
    dims = (4, 4, 4, 4)
    U = np.zeros((256, 4, 3, 3), np.complex128)
    U[:] = np.eye(3)
    U[37, 2] = O.gen_hot(dims, 5)[0, 0]
    _check(dims, U, "fp64", 1e-11, mag=0, n_stout=2, rho=0.1)


@pytest.mark.parametrize("n_stout", [0, 2])
def test_force_is_the_same_bits_alone_and_beside_a_larger_chain(n_stout):
    """Up to 148 tiles (4736 sites) the FP64 plaquette kernels run one block per SM with more
    registers: the same bits as in a larger context."""
    dims = (8, 8, 8, 8)
    U = O.gen_hot(dims, 13)
    with M.Chmc(dims, mag=2, n_stout=n_stout) as s, \
            M.Chmc(chains=[dict(dims=dims), dict(dims=(6, 6, 6, 4))], mag=2, n_stout=n_stout) as e:
        s.set_gauge(U)
        e.set_gauge(U, chain=0)
        assert np.array_equal(s.get_force(), e.get_force(0))
