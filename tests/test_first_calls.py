"""A context's first calls take what the later ones take where nothing is kept between them."""
import time

import pytest

import mag_b200 as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["avg_plaquette", "gauge_action", "kinetic_energy"])
def test_first_measurement_allocates_nothing(call):
    """Fastest first call of contexts made one after another (each closed before the next), in ms: up to
    50, so that a host that is busy for a moment does not decide.  A call is 0.02 to 0.1 ms; with
    the pinned result block's allocation inside 1.4 to 6 ms."""
    best = 1e9
    for _ in range(50):
        with M.Chmc((4, 4, 4, 8), mag=2) as c:
            c.hot_start(3)
            c.init_momentum(traj=0)
            t = time.perf_counter()
            getattr(c, call)()
            best = min(best, 1e3 * (time.perf_counter() - t))
        if best < 0.7:
            break
    assert best < 0.7
