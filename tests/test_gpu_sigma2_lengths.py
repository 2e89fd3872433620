"""Every transform length of the Sigma2 kernels, both as N1 and as N2, against the oracle (whose
own padded length is the reference's): grids of L^2 / 2 energies take the split L x L."""
import numpy as np
import pytest

import oracle_lib
import quichotte_b200 as qb

pytestmark = pytest.mark.gpu
LENGTHS = [16, 20, 24, 28, 32, 36, 40, 48, 56, 64, 72, 80, 96, 112, 128, 144, 160, 192, 224, 256]


def helix(n, U=(0.9, 0.9, 0.9)):
    m = qb.Model.helix(N_ions=3, N_turns=1, hel_length=1.0, hel_radius=0.7, hand=1.0, E_CC=0.0, t_hop=1.0, lamb=0.05,
                       U_int=0.9, GammaL_up=0.6, GammaL_down=0.4, GammaR=0.5, T=300.0, mu=0.1, dw=2.0, up=2.0,
                       delta=0.5, order=2)
    m.U_site[0::2] = U
    m.n_omega, m.delta = n, 8.0 / n
    m.omega = -4.0 + m.delta * np.arange(1, n + 1)
    return m


def errors(m, precision):
    gs, os_ = qb.Solver(m, precision=precision), oracle_lib.solver(m)
    assert gs.Nf == os_.Nf and gs.nA == os_.nA
    x = os_.initial_vector(0.3)
    x = x + 1e-3 * np.random.default_rng(5).standard_normal(x.size)
    rel = lambda a, b: np.max(np.abs(a - b)) / np.max(np.abs(b))
    (SR, SL, S1), (SRo, SLo, S1o) = gs.self_energies(x), os_.self_energies(x)
    return rel(SR, SRo), rel(SL, SLo), rel(S1, S1o)


# FP64: as the transforms' other tests; FP32: rounding relative to the largest spectrum
@pytest.mark.parametrize("L", LENGTHS)
@pytest.mark.parametrize("precision, tol", [(qb.QS_PREC_FP64, 1e-12), (qb.QS_PREC_MIXED, 2e-5)])
def test_every_length_matches_oracle(L, precision, tol):
    eR, eL, e1 = errors(helix(L * L // 2), precision)
    assert eR < tol and eL < tol and e1 < 1e-12, (eR, eL, e1)


@pytest.mark.parametrize("n", [1, 2, 37, 129, 1000, 2001])
def test_padding_and_sites_without_interaction(n):
    # an odd remainder of the split, and a site pair table with holes (U = 0 on the middle site,
    # which then is no active site, and on the first, which its lead keeps active)
    for U in ((0.9, 0.0, 0.4), (0.0, 0.7, 0.4)):
        eR, eL, e1 = errors(helix(n, U), qb.QS_PREC_FP64)
        assert eR < 1e-12 and eL < 1e-12 and e1 < 1e-12, (n, U, eR, eL, e1)
