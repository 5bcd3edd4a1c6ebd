"""Planar Wilson loops in the temporal gauge (k_wloop_gauged) at the edges of its shapes, and the
line products that links and extents outside them still take, against the oracle's loops.

Bar: a loop is a product of at most 2 (R + T) links and 4 Lt gauge factors, each product rounding
at 1e-15; the averages are compared at 1e-12 (general path: as test_wilson_loops_parity).
"""
import numpy as np
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu


def _compare(c, dims, U, R, T, chain=0):
    W = c.wilson_loops(R, T, chain=chain)
    for r in {1, 2, R}:
        for t in {1, T // 2 + 1, T}:
            if r <= R and t <= T:
                ref = O.wilson_loop(dims, U, (r, 0, 0), t)
                assert abs(W[r - 1, t - 1] - ref) < 1e-12 * max(1.0, abs(ref)), (r, t)


@pytest.mark.parametrize("dims,R,T", [
    ((4, 4, 4, 6), 3, 6),       # T = Lt: every loop of that length crosses the boundary
    ((3, 5, 3, 9), 4, 9),       # spatial sites off the block width, slices off the groups, T over one chunk
    ((2, 2, 2, 2), 3, 2),       # R beyond the extent
    ((4, 2, 2, 34), 2, 17),     # several chunks of T
    ((2, 2, 2, 130), 1, 5),     # few sites per block
    ((4, 4, 4, 4), 2, 7),       # T > Lt: line products
])
def test_loops_against_the_oracle(dims, R, T):
    U = O.gen_hot(dims, 17)
    with M.Chmc(dims, mag=0) as c:
        c.set_gauge(U)
        _compare(c, dims, U, R, T)


def test_links_that_are_not_unitary_take_the_line_products():
    dims = (4, 4, 4, 6)
    U = O.gen_hot(dims, 18)
    U[5, 3] *= 1.01
    V = O.gen_hot(dims, 18)
    V[7, 1] *= 1.01
    with M.Chmc(dims, mag=0) as c:
        for A in (U, V):
            c.set_gauge(A)
            _compare(c, dims, A, 3, 4)


@pytest.mark.parametrize("dims,T", [((4, 4, 4, 6), 4), ((4, 4, 4, 6), 6), ((10, 10, 10, 16), 3), ((10, 10, 10, 17), 5)])
def test_unitary_links_of_any_determinant(dims, T):
    """Antiperiodic time links, and a U(1) phase on time and spatial links: unitary, not special.
    On both sides of the line between one and two slices per thread."""
    U = O.gen_hot(dims, 21)
    U[-dims[0] * dims[1] * dims[2]:, 3] *= -1
    V = O.gen_hot(dims, 22)
    V *= np.exp(1j * np.random.default_rng(3).uniform(-1, 1, V.shape[:2]))[..., None, None]
    with M.Chmc(dims, mag=0) as c:
        for A in (U, V):
            c.set_gauge(A)
            _compare(c, dims, A, 3, T)


@pytest.mark.parametrize("dims,T", [((4, 4, 4, 6), 6), ((4, 4, 4, 24), 9)])
def test_links_that_drifted_off_unitarity_keep_their_loops(dims, T):
    """Links of one gauge orbit (every loop 1) times 1 + e H with e = 1e-13, H Hermitian of order one:
    a loop of 2 (R + T) of them is off one by some 1e-12, none of which may be lost.

    Bar: the products of a loop's own links and of its gauge factors, 2 (R + T) + 4 Lt of them, round
    by at most 4 * 2^-53 per element, three of which enter the trace (a loop of unit links is 3).
    They are of random sign, on 3 V loops that are averaged; a tenth of their sum is asked.
    """
    V = int(np.prod(dims))
    rng = np.random.default_rng(6)
    x = O.gen_hot(dims, 23)[:, 0].reshape(dims[::-1] + (3, 3))
    U = np.empty(dims[::-1] + (4, 3, 3), np.complex128)
    for mu in range(4):
        U[..., mu, :, :] = x @ np.roll(x, -1, axis=3 - mu).conj().swapaxes(-1, -2)
    U = U.reshape(V, 4, 3, 3)
    A = rng.standard_normal(U.shape) + 1j * rng.standard_normal(U.shape)
    H = (A + A.conj().swapaxes(-1, -2)) / 8 + 0.5 * np.eye(3)
    U = U + 1e-13 * (H @ U)
    with M.Chmc(dims, mag=0) as c:
        c.set_gauge(U)
        W = c.wilson_loops(2, T)
    for r, t in ((1, 1), (2, 2), (2, T)):
        assert abs(W[r - 1, t - 1] - O.wilson_loop(dims, U, (r, 0, 0), t)) <= 12 * 2.0**-53 * (2 * (r + t) + 4 * dims[3]) / 10


@pytest.mark.parametrize("dims,R,T", [((2, 2, 2, 300), 2, 5), ((4, 4, 6, 201), 2, 4), ((6, 5, 6, 97), 2, 8),
                                      ((8, 8, 8, 33), 2, 4)])
def test_two_slices_per_thread_and_an_odd_number_of_slots(dims, R, T):
    """One, two, four and eight spatial sites per block; Lt + Tmax odd, so that the last slot of the second
    slices stays empty; Lt odd, so that the last thread has one slice."""
    U = O.gen_hot(dims, 24)
    with M.Chmc(dims, mag=0) as c:
        c.set_gauge(U)
        _compare(c, dims, U, R, T)


def test_one_chain_of_an_ensemble():
    dims = [(4, 4, 4, 4), (2, 4, 4, 6)]
    with M.Chmc(chains=[dict(dims=d) for d in dims], mag=2) as c:
        Us = [O.gen_hot(d, 20 + k) for k, d in enumerate(dims)]
        for k, U in enumerate(Us):
            c.set_gauge(U, chain=k)
        for k, U in enumerate(Us):
            _compare(c, dims[k], U, 2, 3, chain=k)
            assert abs(c.avg_plaquette(k) - O.avg_plaquette(dims[k], U)) < 1e-14
