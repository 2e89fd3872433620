"""The sums over energies at the edges of their split over blocks (rows per thread, blocks per
column group), through an order-0 IV point against the oracle."""
import numpy as np
import pytest

import oracle_lib
import quichotte_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sites", [(4, 1), (5, 7)])
@pytest.mark.parametrize("n", [1, 7, 128, 129, 2047, 2049, 8193])
def test_sums_over_energies_match_oracle(sites, n):
    m = qb.Model.helix(N_ions=sites[0], N_turns=sites[1], hel_length=1.0, hel_radius=0.7, hand=1.0, E_CC=0.0, t_hop=1.0,
                       lamb=0.05, U_int=0.0, GammaL_up=0.6, GammaL_down=0.4, GammaR=0.5, T=300.0, mu=0.1, dw=1.0,
                       up=1.0, delta=0.5, order=0)
    m.n_omega, m.delta = n, 6.0 / n
    m.omega = -3.0 + m.delta * np.arange(1, n + 1)
    g, o = qb.Solver(m), oracle_lib.solver(m)
    g.solve_scf(0.3, True), o.solve_scf(0.3, True)
    a, b = g.observables(), o.observables()
    # n rounded additions of terms computed to a few ulps of the largest inverse element
    tol = 1e-12 * max(1.0, np.max(np.abs(b["dosd"])))
    for k in ("G_less_obs", "dosd", "trU", "trD"):
        assert np.max(np.abs(a[k] - b[k])) <= tol, k
    assert np.max(np.abs(np.array(g.current(0.3)) - o.current(0.3))) <= tol
