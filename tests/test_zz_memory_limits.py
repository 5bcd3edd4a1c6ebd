"""Calls that need less device memory by an older form still succeed where the faster form's
fields are not to be had.  Each test takes most of the device's memory with one allocation of its
own and gives it back.  Collected last: a stop-at-first-failure run has then run every other test.
"""
import numpy as np
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu

MB = 1 << 20


class leave:
    """Leaves about `mb` MB of the device's memory free."""

    def __init__(self, mb):
        self.mb = mb

    def __enter__(self):
        import torch

        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.held = torch.empty(free - self.mb * MB, dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch

        self.held = None
        torch.cuda.empty_cache()


@pytest.mark.parametrize("left,scaled", [(80, False), (130, True)])
def test_loops_without_room_for_the_temporal_gauge(left, scaled):
    """16^3 x 32: the gauged form takes 104 MB, the line products of one length 57 MB.  With 80 MB left
    they are all that fits; with 130 MB left links that are not unitary are found out by the gauged
    form, whose fields have to make room.  Bar as for the other loops, 1e-12."""
    dims = (16, 16, 16, 32)
    with M.Chmc(dims, mag=0, seed=3) as c:
        c.hot_start(4)
        U = c.get_gauge()
        if scaled:
            U[5, 3] *= 1.01
            c.set_gauge(U)
        with leave(left):
            W = c.wilson_loops(1, 2)
        for t in (1, 2):
            ref = O.wilson_loop(dims, U, (1, 0, 0), t)
            assert abs(W[0, t - 1] - ref) < 1e-12 * max(1.0, abs(ref))
        assert np.abs(c.wilson_loops(2, 2)[0] - W[0]).max() < 1e-12
