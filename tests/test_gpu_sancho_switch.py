"""SANCHO's longest transforms and the step to the direct sums (6720 energies: the longest sequence that fits in
shared memory has 13440 values), against the oracle, as test_gpu_sancho_lengths.py."""
import pytest

from test_gpu_sancho_lengths import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, order", [(6720, 2), (6720, 3), (6721, 2)])
def test_both_sides_of_the_longest_transform(tmp_path, n, order):
    compare(tmp_path, n, order, 2)
