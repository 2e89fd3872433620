"""An infinite pivot: below order 16, and in qs_invert_batched_noalloc at every order, its reciprocal is 0 and the
other states are untouched, as the elimination by Smith's division gives it."""
import numpy as np
import pytest

import quichotte_b200 as qb
from test_zz_no_alloc import run_noalloc

pytestmark = pytest.mark.gpu
VALUES = [complex(np.inf, 0.5), complex(-np.inf, 0.5), complex(0.5, np.inf)]


def case(N, value):
    d = np.arange(1.0, N + 1) + 0.5j
    A = np.zeros((2, N, N), np.complex128)
    A[:, range(N), range(N)] = d
    A[1, N // 2, N // 2] = value
    ref = np.array([np.diag(1.0 / d)] * 2)
    ref[1, N // 2, N // 2] = 0.0
    return A, ref


@pytest.mark.parametrize("N", [1, 2, 8, 9, 15])
@pytest.mark.parametrize("value", VALUES)
def test_infinite_pivot(N, value):
    A, ref = case(N, value)
    inv, info = qb.invert_batched(A)
    assert not info.any() and np.max(np.abs(inv - ref)) < 1e-15


@pytest.mark.parametrize("N, copies", [(1, 1), (9, 1), (16, 1), (40, 1), (80, 1), (96, 1), (120, 1), (120, 80), (121, 1), (200, 1),
                                       (260, 1)])
@pytest.mark.parametrize("value", VALUES)
def test_infinite_pivot_without_allocation(N, copies, value):
    torch = pytest.importorskip("torch")
    A, ref = case(N, value)
    inv, info = run_noalloc(torch, np.tile(A, (copies, 1, 1)))
    assert not info.any() and np.max(np.abs(inv - np.tile(ref, (copies, 1, 1)))) < 1e-15
