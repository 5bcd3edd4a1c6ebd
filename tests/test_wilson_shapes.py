"""Wilson loops in the temporal gauge on both sides of the shape line (one slice per thread for
few sites, three for more) and of the trace chunk (T <= 4 or more), against the oracle's loops.

Bar: as for the other loops of this path, products of at most 2 (R + T) links and 4 Lt gauge
factors rounding at 1e-15 each: 1e-12.
"""
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R,T", [
    ((4, 4, 4, 9), 2, 4),        # one slice per thread, one chunk of four
    ((4, 4, 4, 9), 2, 5),        # chunk of eight
    ((11, 10, 9, 32), 3, 4),     # 32,670 threads of three slices, the last group short
    ((11, 10, 9, 31), 2, 9),     # the same, two chunks of eight
    ((10, 10, 10, 30), 2, 3),    # exactly at the line
    ((10, 10, 10, 27), 2, 3),    # below it
    ((2, 2, 2, 260), 1, 3),      # more slices than threads: three per thread
])
def test_loops_across_the_shapes(dims, R, T):
    U = O.gen_hot(dims, 19)
    with M.Chmc(dims, mag=0) as c:
        c.set_gauge(U)
        W = c.wilson_loops(R, T)
    for r, t in {(1, 1), (R, 1), (1, T), (R, T)}:
        ref = O.wilson_loop(dims, U, (r, 0, 0), t)
        assert abs(W[r - 1, t - 1] - ref) < 1e-12 * max(1.0, abs(ref)), (r, t)
