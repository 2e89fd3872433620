"""The SCF residual above 80 states, at the orders where the Dyson and Keldysh kernels change their shape
(blocks of 32 rows, row tiles of 16, column tiles of 8, the step to the general kernels), against the
oracle, with and without x subtracted (the fresh-start vector), FP64."""
import pytest

from test_gpu_keldysh_orders import residual_errors

pytestmark = pytest.mark.gpu
# sites per turn x turns; order = 2 x sites
HELICES = [(41, 1), (11, 4), (12, 4), (7, 7), (14, 4), (10, 6), (61, 1), (9, 7), (16, 4), (13, 5), (20, 4), (12, 8),
           (97, 1), (16, 7), (113, 1), (127, 1), (16, 8), (43, 3)]


# as the other residual tests: FP64 rounding times the conditioning of the Dyson matrices
@pytest.mark.parametrize("ions, turns", HELICES)
def test_residual_matches_oracle(ions, turns):
    for n in (1, 9):
        e0, e1 = residual_errors(ions, turns, n)
        assert e0 < 1e-11 and e1 < 1e-11, (n, e0, e1)


@pytest.mark.parametrize("ions, turns, contacts", [(11, 4, 3), (12, 4, 20), (13, 5, 15), (12, 8, 32)])
def test_dense_lead_matrices(ions, turns, contacts):
    e0, e1 = residual_errors(ions, turns, 11, contacts)
    assert e0 < 1e-11 and e1 < 1e-11, (e0, e1)
