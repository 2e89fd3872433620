"""Order-2 residuals and outputs of models whose active states are few: the Dyson matrices are larger than G_AA, so
that they are inverted in shared memory up to order 120 and above it in the slots of a workspace, more energies than
slots, against the oracle."""
import numpy as np
import pytest

import oracle_lib
import quichotte_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ions, turns, n", [(3, 3, 20), (9, 4, 30), (11, 4, 160), (10, 6, 9), (61, 1, 310), (16, 7, 5), (43, 3, 4)])
def test_inactive_states_match_oracle(ions, turns, n):
    m = qb.Model.helix(N_ions=ions, N_turns=turns, hel_length=0.3 * turns, hel_radius=0.7, hand=1.0, E_CC=0.0, t_hop=1.0, lamb=0.01,
                       U_int=0.7, GammaL_up=0.5, GammaL_down=0.4, GammaR=0.5, T=300.0, mu=0.0, dw=1.0, up=1.0, delta=0.5, order=2)
    U = np.zeros(m.Norb)
    U[4:8] = U[-10:-6] = 0.7  # four interacting sites, and the contacts
    m.U_site = U
    m.n_omega, m.delta = n, 6.0 / n
    m.omega = -3.0 + m.delta * np.arange(1, n + 1)
    g, o = qb.Solver(m, maxscf=1), oracle_lib.solver(m, maxscf=1)
    assert 0 < g.nA < m.Norb
    xg, xo = g.initial_vector(0.3), o.initial_vector(0.3)
    x = xo + 1e-3 * np.random.default_rng(2).standard_normal(xo.size)
    (Fg, ag), (Fo, ao) = g.residual(0.3, x), o.residual(0.3, x)
    assert ag == ao
    # as the other residual tests: FP64 rounding times the conditioning of the Dyson matrices
    scale = max(1.0, np.max(np.abs(x)), np.max(np.abs(Fo)))
    assert np.max(np.abs(xg - xo)) < 1e-11 * scale and np.max(np.abs(Fg - Fo)) < 1e-11 * scale
    out = []
    for sol in (g, o):
        sol.solve_scf(0.3, True)
        out.append(dict(sol.observables(), current=np.atleast_1d(np.array(sol.current(0.3)))))
    for k, ref in out[1].items():
        assert np.max(np.abs(np.asarray(out[0][k]) - ref)) < 1e-11 * max(1.0, np.max(np.abs(ref))), k
