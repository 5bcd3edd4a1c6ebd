"""Per-link demon sweep where neighbouring links overlap (every extent >= 5, so that the
site offsets -2..2 are distinct) and where they do not, on both sides of that line, against
the oracle's sequential restatement (demon_microcanonical, field-demon.h:25-126).

Bars as for the other sweeps: identical hit counts, demon energies within 1e-9 (sums of
O(1) action changes over thousands of hits), swept links within 1e-12.
"""
import numpy as np
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(5, 5, 5, 5), (5, 6, 7, 5), (7, 5, 5, 6), (4, 5, 6, 5), (5, 5, 3, 5), (5, 5, 5, 2)])
def test_sweeps_match_oracle_across_the_overlap_line(dims):
    U = O.gen_hot(dims, 13)
    Uo, Eo, ao, ro, _ = O.demon_sweeps(dims, U, seed=17, n_sweeps=2, e_max=12.0)
    with M.Chmc(dims, mag=0) as c:
        c.set_gauge(U)
        res = c.demon_microcanonical(2, 12.0, seed=17, update_links=True)
        Ug = c.get_gauge()
    assert res["accepted"] == ao and res["rejected"] == ro
    assert ao > 0 and ro > 0
    assert np.abs(res["demon_energy"] - Eo).max() < 1e-9
    assert np.abs(Ug - Uo).max() < 1e-12
