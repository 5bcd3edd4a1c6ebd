"""The Wilson action's force through smeared links and the fused uses of a force (momentum kick, link
update of the force-gradient step), in both precisions, against the oracle.

Bars: the parity bars of test_gpu_parity.py.  Forces 1e-11 of the largest component in FP64 and
5e-5 mixed; a trajectory's Delta H 1e-9 + 1e-11 |Delta H| and its links 1e-10 in FP64, Delta H 5e-3 +
2e-3 |Delta H| and the plaquette 1e-7 mixed, with the same accept decision.
"""
import numpy as np
import pytest

import mag_b200 as M
import oracle as O

pytestmark = pytest.mark.gpu

FORCE_BAR = {"fp64": 1e-11, "mixed": 5e-5}


@pytest.mark.parametrize("precision", list(FORCE_BAR))
@pytest.mark.parametrize("dims,mag,n_stout,rho", [
    ((4, 4, 4, 8), 2, 0, 0.1), ((5, 3, 3, 4), 0, 0, 0.1), ((5, 3, 3, 4), 0, 1, 0.1), ((5, 3, 3, 4), 0, 2, 0.1),
    ((2, 2, 2, 2), 2, 1, 0.1), ((2, 6, 4, 3), 0, 3, 0.1), ((4, 4, 4, 4), 2, 2, 0.8), ((8, 4, 4, 8), 4, 1, 0.1),
    ((3, 4, 5, 2), 0, 1, 3.0)])
def test_wilson_force(dims, mag, n_stout, rho, precision):
    """Partial tiles, extents of two, exponents beyond the series of Lambda."""
    U = O.gen_hot(dims, 11)
    F0 = O.force(O.make_params(dims, mag=mag, action=0, beta=5.6, n_stout=n_stout, rho=rho), U)
    with M.Chmc(dims, action="wilson", beta=5.6, mag=mag, n_stout=n_stout, rho=rho, precision=precision) as c:
        c.set_gauge(U)
        F = c.get_force()
    assert np.abs(F - F0).max() < FORCE_BAR[precision] * max(1.0, np.abs(F0).max())


@pytest.mark.parametrize("precision", list(FORCE_BAR))
def test_wilson_force_of_an_ensembles_chains(precision):
    dims, kw = [(4, 4, 4, 4), (5, 3, 3, 4), (2, 4, 6, 2)], dict(mag=0, n_stout=2, rho=0.1)
    with M.Chmc(chains=[dict(dims=d, beta=5.5 + 0.1 * k) for k, d in enumerate(dims)], action="wilson",
                precision=precision, **kw) as c:
        U = [O.gen_hot(d, 12 + k) for k, d in enumerate(dims)]
        for k in range(3):
            c.set_gauge(U[k], chain=k)
        for k, d in enumerate(dims):
            F0 = O.force(O.make_params(d, action=0, beta=5.5 + 0.1 * k, **kw), U[k])
            assert np.abs(c.get_force(k) - F0).max() < FORCE_BAR[precision] * max(1.0, np.abs(F0).max())


@pytest.mark.parametrize("precision", list(FORCE_BAR))
@pytest.mark.parametrize("dims,action,mag,n_stout,integrator", [
    ((4, 4, 4, 8), "wilson", 2, 0, "fg"), ((4, 4, 4, 8), "wilson", 2, 0, "leapfrog"),
    ((4, 6, 4, 5), "wilson", 0, 2, "leapfrog"), ((4, 4, 4, 8), "wilson", 2, 1, "fg"),
    ((8, 4, 4, 8), "wilson", 4, 0, "fg"), ((8, 4, 4, 8), "iwasaki", 4, 0, "fg"),
    ((8, 4, 4, 8), "iwasaki", 4, 2, "fg"), ((6, 6, 3, 6), "iwasaki", 3, 1, "fg")])
def test_trajectory_by_the_fused_uses(dims, action, mag, n_stout, integrator, precision):
    """mag = 3 and 4: segments whose inner links move with the force of the link before them too."""
    kw = dict(mag=mag, n_stout=n_stout, rho=0.1, beta=5.6 if action == "wilson" else 2.25, n_steps=12)
    po = O.make_params(dims, action=1 if action == "iwasaki" else 0, integrator=1 if integrator == "leapfrog" else 0, **kw)
    U, P, u = O.gen_hot(dims, 14), O.gen_momenta(dims, 6, 0), O.gen_uniform(6, 0)
    with M.Chmc(dims, action=action, integrator=integrator, precision=precision, seed=6, **kw) as c:
        c.set_gauge(U)
        c.init_momentum(P)
        c.set_uniforms([u])
        (g,) = c.trajectory(refresh_momenta=False)
        Ug = c.get_gauge()
    Uo, o = O.trajectory(po, 0, U, P, u, [0.0, 0.0])
    assert g["accept"] == o["accept"]
    if precision == "fp64":
        assert abs(g["delta_h"] - o["delta_h"]) < 1e-9 + 1e-11 * abs(o["delta_h"])
        assert np.abs(Ug - Uo).max() < 1e-10
    else:
        assert abs(g["delta_h"] - o["delta_h"]) < 5e-3 + 2e-3 * abs(o["delta_h"])
        assert abs(g["avg_plaquette"] - o["avg_plaquette"]) < 1e-7


def test_loops_of_links_moved_without_reunitarisation():
    """Leapfrog steps leave the links off unitarity by the roundings of their updates; their loops are
    those of the links as they are (bar of the other loops, 1e-12)."""
    dims = (4, 4, 4, 12)
    with M.Chmc(dims, mag=0, n_stout=1, integrator="leapfrog", n_steps=30, seed=4) as c:
        c.hot_start(5)
        for k in range(5):
            c.init_momentum(traj=k)
            c.force_gradient_integrator()
        U, W = c.get_gauge(), c.wilson_loops(2, 12)
    assert np.abs(U @ U.conj().swapaxes(-1, -2) - np.eye(3)).max() > 1e-15
    for r, t in ((1, 1), (2, 3), (1, 12), (2, 12)):
        assert abs(W[r - 1, t - 1] - O.wilson_loop(dims, U, (r, 0, 0), t)) < 1e-12
