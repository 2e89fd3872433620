"""Solves at several voltages on one handle, whose captured steps serve all of them, against solves on handles of
their own (bit for bit), with odd and even step counts (the buffers change places)."""
import numpy as np
import pytest

import quichotte_b200 as qb

pytestmark = pytest.mark.gpu


def run(s, V):
    r = s.solve_scf(V, True)
    return dict(s.observables(), J=np.array(s.current(V)), n=r["n_iter"], fmax=r["fmax"])


@pytest.mark.parametrize("ions, turns", [(4, 1), (11, 4)])
@pytest.mark.parametrize("steps", [4, 5])
def test_one_handle_many_voltages(ions, turns, steps):
    m = qb.Model.helix(N_ions=ions, N_turns=turns, hel_length=0.3 * turns, hel_radius=0.7, hand=1.0, E_CC=0.0, t_hop=1.0,
                       lamb=0.01, U_int=0.7, GammaL_up=0.5, GammaL_down=0.4, GammaR=0.5, T=300.0, mu=0.0, dw=1.0, up=1.0,
                       delta=0.5, order=2)
    m.n_omega, m.delta = 61, 0.1
    m.omega = -3.0 + m.delta * np.arange(1, 62)
    one = qb.Solver(m, maxscf=steps, tolf=1e-14)
    for V in (0.3, -0.2, 0.3, 0.7, 0.0, -0.0):
        a, own = run(one, V), qb.Solver(m, maxscf=steps, tolf=1e-14)
        b = run(own, V)
        own.close()
        for k in b:
            assert np.array_equal(a[k], b[k]), (V, k)
    assert one.graph_replays() > 0
