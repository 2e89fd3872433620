"""The final sweep of order-2 models with few active states: its chunks of full matrices fill the device, whatever the
number of active states (a launch of the inversion and one of the outputs each)."""
import numpy as np
import pytest

import quichotte_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ions, turns, n", [(10, 6, 200), (10, 6, 1000), (12, 8, 500)])
def test_few_active_states_take_few_launches(ions, turns, n):
    m = qb.Model.helix(N_ions=ions, N_turns=turns, hel_length=0.3 * turns, hel_radius=0.7, hand=1.0, E_CC=0.0, t_hop=1.0, lamb=0.01,
                       U_int=0.7, GammaL_up=0.5, GammaL_down=0.4, GammaR=0.5, T=300.0, mu=0.0, dw=1.0, up=1.0, delta=0.5, order=2)
    U = np.zeros(m.Norb)
    U[4:6] = 0.7
    m.U_site = U
    m.n_omega, m.delta = n, 6.0 / n
    m.omega = -3.0 + m.delta * np.arange(1, n + 1)
    s = qb.Solver(m, maxscf=1)
    before = qb._lib.qs_kernel_launches()
    s.solve_scf(0.3, True)
    # start, one step, the sums: 20; two for each chunk of at least 256 energies
    assert qb._lib.qs_kernel_launches() - before <= 20 + 2 * (-(-n // 256))
