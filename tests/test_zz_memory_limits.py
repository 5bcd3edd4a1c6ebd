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


@pytest.mark.parametrize("kw,left", [(dict(), 2450), (dict(n_stout=2, precision="mixed"), 4170)])
def test_contexts_without_room_for_the_plaquette_form(kw, left):
    """24^3 x 48: thin FP64 takes 2.25 GB without the plaquette form's fields and 2.93 GB with them,
    mixed with two levels 4.25 and 4.50 GB.  Forces as in test_gpu_parity.py, 1e-11 FP64 and 5e-5 mixed;
    the Hamiltonian (FP64) within 1e-12."""
    dims = (24, 24, 24, 48)
    kw = dict(kw, mag=2, n_steps=1, seed=9)

    def measure(c):
        c.hot_start(4)
        c.init_momentum(traj=0)
        F, h = c.get_force(), c.get_hamiltonian()[0]
        (rec,) = c.trajectory()
        return c.device_bytes(), F, h, rec

    with M.Chmc(dims, **kw) as c:
        b0, F0, h0, r0 = measure(c)
    with leave(left):
        with M.Chmc(dims, **kw) as c:
            b1, F1, h1, r1 = measure(c)
            with pytest.raises(M.MagError):
                c.time_kernel("plaq_force", 1)
    assert b1 < left * MB < b0
    assert np.abs(F1 - F0).max() < (5e-5 if "precision" in kw else 1e-11) * max(1.0, np.abs(F0).max())
    assert abs(h1 - h0) <= 1e-12 * abs(h0) and r1["accept"] == r0["accept"]


def test_shards_without_room_for_the_plaquette_form():
    """Two thin FP64 slabs of 16^3 x 64, each 32 slices and a halo of two on both sides: 3392 bytes per
    site without the plaquette form's fields and 4416 with them, 1.00 and 1.30 GB in all."""
    from mag_b200.dd import DomainChmc

    dims = (16, 16, 16, 64)
    with DomainChmc(dims, 2, mag=2) as d:
        d.hot_start(4)
        F0 = d.get_force()
    with leave(1100):
        with DomainChmc(dims, 2, mag=2) as d:
            d.hot_start(4)
            F1 = d.get_force()
    assert np.abs(F1 - F0).max() < 1e-11 * np.abs(F0).max()
