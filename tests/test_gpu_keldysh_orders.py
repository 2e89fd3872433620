"""The SCF residual over the orders at which the Dyson and Keldysh kernels change their shape (row
tiles of 16, column tiles of 8, warps per matrix), against the oracle, with and without x subtracted
(the fresh-start vector), FP64."""
import numpy as np
import pytest

import oracle_lib
import quichotte_b200 as qb

pytestmark = pytest.mark.gpu
# sites per turn x turns; nA = 2 x sites
HELICES = [(2, 1), (3, 1), (4, 1), (5, 1), (3, 3), (5, 2), (4, 3), (13, 1), (4, 4), (17, 1), (5, 4), (7, 3), (6, 4),
           (7, 4), (8, 4), (11, 3), (9, 4), (37, 1), (8, 5)]


def residual_errors(ions, turns, n, contacts=None):
    m = qb.Model.helix(N_ions=ions, N_turns=turns, hel_length=0.3 * turns, hel_radius=0.7, hand=1.0, E_CC=0.0, t_hop=1.0,
                       lamb=0.01, U_int=0.7, GammaL_up=0.5, GammaL_down=0.4, GammaR=0.5, T=300.0, mu=0.0, dw=1.0, up=1.0,
                       delta=0.5, order=2)
    if contacts:  # dense lead matrices on the first and last `contacts` states
        rng = np.random.default_rng(1)
        for G, s in ((m.GammaL, slice(0, contacts)), (m.GammaR, slice(m.Norb - contacts, m.Norb))):
            A = rng.standard_normal((contacts, contacts)) + 1j * rng.standard_normal((contacts, contacts))
            G[s, s] += 0.02 * (A @ A.conj().T)
    m.n_omega, m.delta = n, 6.0 / n
    m.omega = -3.0 + m.delta * np.arange(1, n + 1)
    g, o = qb.Solver(m), oracle_lib.solver(m)
    assert g.nA == m.Norb
    xg, xo = g.initial_vector(0.3), o.initial_vector(0.3)
    x = xo + 1e-3 * np.random.default_rng(2).standard_normal(xo.size)
    (Fg, ag), (Fo, ao) = g.residual(0.3, x), o.residual(0.3, x)
    assert ag == ao
    scale = max(1.0, np.max(np.abs(x)), np.max(np.abs(Fo)))
    return np.max(np.abs(xg - xo)) / scale, np.max(np.abs(Fg - Fo)) / scale


# as the other residual tests: FP64 rounding times the conditioning of the Dyson matrices
@pytest.mark.parametrize("ions, turns", HELICES)
def test_residual_matches_oracle(ions, turns):
    for n in (1, 150):  # a single energy, and more than one per SM
        e0, e1 = residual_errors(ions, turns, n)
        assert e0 < 1e-11 and e1 < 1e-11, (n, e0, e1)


@pytest.mark.parametrize("ions, turns, contacts", [(3, 2, 3), (6, 4, 20)])
def test_dense_lead_matrices(ions, turns, contacts):
    e0, e1 = residual_errors(ions, turns, 37, contacts)
    assert e0 < 1e-11 and e1 < 1e-11, (e0, e1)
