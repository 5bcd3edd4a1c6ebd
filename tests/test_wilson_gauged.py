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


def test_one_chain_of_an_ensemble():
    dims = [(4, 4, 4, 4), (2, 4, 4, 6)]
    with M.Chmc(chains=[dict(dims=d) for d in dims], mag=2) as c:
        Us = [O.gen_hot(d, 20 + k) for k, d in enumerate(dims)]
        for k, U in enumerate(Us):
            c.set_gauge(U, chain=k)
        for k, U in enumerate(Us):
            _compare(c, dims[k], U, 2, 3, chain=k)
            assert abs(c.avg_plaquette(k) - O.avg_plaquette(dims[k], U)) < 1e-14
