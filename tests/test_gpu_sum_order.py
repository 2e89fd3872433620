"""The order of the sums over energies at first order, where the on-site sums of G^< are the SCF vector itself and
sharp levels turn its last bits into 1e-10 of the spectra: eight chains over the energies 0..7 (mod 8), added one
after the other, for every grid. Equal bits, without a tolerance."""
import numpy as np
import pytest

import quichotte_b200 as qb

pytestmark = pytest.mark.gpu


def model(ions, turns, n, order, U):
    m = qb.Model.helix(N_ions=ions, N_turns=turns, hel_length=1.0, hel_radius=0.7, hand=1.0, E_CC=0.0, t_hop=1.0, lamb=0.05,
                       U_int=U, GammaL_up=0.6, GammaL_down=0.4, GammaR=0.5, T=300.0, mu=0.1, dw=1.0, up=1.0, delta=0.5,
                       order=order)
    m.n_omega = n
    m.delta = 2.0 * np.pi / 64  # delta / 2 pi is a power of two: no further rounding
    m.omega = -0.5 * n * m.delta + m.delta * np.arange(1, n + 1)
    return m


def in_order(v):
    """Sums over axis 0."""
    chains = [np.cumsum(v[l::8], axis=0)[-1] if l < len(v) else np.zeros_like(v[0]) for l in range(8)]
    return np.cumsum(chains, axis=0)[-1]


# below eight energies, one tile of 128 and its edges, more tiles than are under way; 8 and 12 columns
@pytest.mark.parametrize("ions, turns, n", [(2, 1, 5), (2, 1, 127), (2, 1, 129), (3, 1, 128), (3, 1, 643)])
def test_first_order_vector_is_the_sum_of_its_energies(ions, turns, n):
    m = model(ions, turns, n, 1, 0.4)
    x = np.zeros(qb.Solver(m).n_vec)
    F, _ = qb.Solver(m).residual(0.3, x)
    each = []
    for w in m.omega:  # a grid of that energy alone
        one = model(ions, turns, 1, 1, 0.4)
        one.omega = np.array([w])
        each.append(qb.Solver(one).residual(0.3, x)[0])
    assert np.array_equal(F, in_order(np.array(each)))
