"""SANCHO's self-energies over the grid lengths at which their transforms change: two, three and four
passes, every radix, the shortest grids, and the step to the direct sums where a sequence no longer fits
in shared memory, against the oracle's direct sums. 1e-11 of the largest element as in test_gpu_sancho.py
(a chain of transforms adds a few rounding errors of the norm each)."""
import numpy as np
import pytest

import oracle_lib
from test_gpu_sancho import case_dir, noisy_input, rel

pytestmark = pytest.mark.gpu

sb = pytest.importorskip("sancho_b200")

GRIDS = [1, 2, 3, 8, 9, 13, 25, 33, 57, 91, 113, 128, 129, 245, 251, 500, 883, 1023, 1499, 2048, 2049, 3000]


def compare(tmp_path, n, order, sites):
    m = sb.SanchoModel.load(case_dir(str(tmp_path), f"n{n}", order=order, N_sites=sites, U_int=0.9))
    m.n_omega, m.delta = n, 4.0 / n
    m.omega = m.delta * np.arange(1, n + 1)
    gs, os_ = sb.SanchoSolver(m), oracle_lib.sancho_solver(m)
    x = noisy_input(os_, 0.25, n)
    for k, (a, b) in enumerate(zip(gs.self_energies(x), os_.self_energies(x))):
        if k < 2 or order == 3:
            assert np.max(np.abs(b)) > 0 and rel(a, b) < 1e-11, (n, k, rel(a, b))


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("order", [2, 3])
def test_self_energies_match_oracle(tmp_path, n, order):
    compare(tmp_path, n, order, 3)


@pytest.mark.parametrize("n, order", [(6700, 2), (6800, 2), (6801, 2), (6801, 3)])
def test_longest_transforms_and_direct_sums(tmp_path, n, order):
    compare(tmp_path, n, order, 2)
