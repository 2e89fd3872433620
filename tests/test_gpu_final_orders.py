"""The outputs of the final sweep (on-site blocks of G^<, Im G^r, the current integrand) over the orders at
which its kernel changes its shape, and for left contacts of one state, of many, and spread over two blocks
of 32 rows (the general kernel), against the oracle, after one SCF step of order 2."""
import numpy as np
import pytest

import oracle_lib
import quichotte_b200 as qb

pytestmark = pytest.mark.gpu
# sites per turn x turns, the states of the left lead, energies
CASES = [(2, 1, (0, 2), 5), (4, 1, (0, 1), 3), (3, 4, (0, 2), 40), (17, 1, (0, 32), 7), (17, 1, (33, 34), 7), (9, 4, (30, 34), 5),
         (11, 3, (40, 44), 6), (10, 6, (0, 2), 9), (13, 5, (64, 80), 4), (12, 8, (0, 2), 3), (16, 8, (254, 256), 2)]


@pytest.mark.parametrize("ions, turns, left, n", CASES)
def test_final_outputs_match_oracle(ions, turns, left, n):
    m = qb.Model.helix(N_ions=ions, N_turns=turns, hel_length=0.3 * turns, hel_radius=0.7, hand=1.0, E_CC=0.0, t_hop=1.0,
                       lamb=0.01, U_int=0.7, GammaL_up=0.5, GammaL_down=0.4, GammaR=0.5, T=300.0, mu=0.0, dw=1.0, up=1.0,
                       delta=0.5, order=2)
    rng = np.random.default_rng(3)
    s = slice(*left)
    A = rng.standard_normal((left[1] - left[0],) * 2) + 1j * rng.standard_normal((left[1] - left[0],) * 2)
    m.GammaL[:] = 0.0
    m.GammaL[s, s] = 0.1 * (A @ A.conj().T) + 0.1 * np.eye(left[1] - left[0])
    m.n_omega, m.delta = n, 6.0 / n
    m.omega = -3.0 + m.delta * np.arange(1, n + 1)
    g, o = qb.Solver(m, maxscf=1), oracle_lib.solver(m, maxscf=1)
    out = []
    for sol in (g, o):
        sol.solve_scf(0.3, True)
        J = np.atleast_1d(np.array(sol.current(0.3)))
        out.append(dict(sol.observables(), current=J))
    for k, ref in out[1].items():
        # as the residual tests: FP64 rounding times the conditioning of the Dyson matrices
        assert np.max(np.abs(np.asarray(out[0][k]) - ref)) < 1e-11 * max(1.0, np.max(np.abs(ref))), k
