"""The batched inversion at the edges of its kernels' orders: panels of 8, warps of 32 rows, the
numbers of warps per matrix (32, 64, 80, 96, 120), the in-place kernels above them (121..256, 257..)."""
import numpy as np
import pytest

import quichotte_b200 as qb

pytestmark = pytest.mark.gpu
ORDERS = [1, 7, 8, 9, 15, 17, 31, 32, 33, 40, 63, 64, 65, 79, 81, 95, 96, 97, 113, 119, 120, 121, 255, 256, 257]


def matrices(N, batch, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((batch, N, N)) + 1j * rng.standard_normal((batch, N, N))


@pytest.mark.parametrize("N", ORDERS)
def test_inverse_matches_numpy(N):
    # enough matrices for several rounds of the small kernels' blocks
    A = matrices(N, 700 if N <= 40 else 9, N) + 3 * np.sqrt(N) * np.eye(N)
    inv, info = qb.invert_batched(A)
    assert not info.any()
    ref = np.linalg.inv(A)
    assert np.max(np.abs(inv - ref)) < 1e-13 * np.max(np.abs(ref))


@pytest.mark.parametrize("N", [5, 16, 40, 77, 120, 121])
def test_pivoting_scaling_and_singular_matrices(N):
    # rows in reverse order with a dominant antidiagonal: every step's pivot lies elsewhere
    A = matrices(N, 6, 7 * N)
    A[0] = 0.01 * A[0] + 3 * np.sqrt(N) * np.eye(N)[::-1]
    well = 0.1 * A[1] + 3 * np.sqrt(N) * np.eye(N)
    A[1], A[2], A[3] = well, well * 1e250, well * 1e-250
    A[4] = well
    A[4][:, N // 2] = 0.0  # a zero column: step N/2 + 1 finds no pivot
    A[5] = 3 * np.sqrt(N) * np.eye(N) + 0.1 * A[5]
    inv, info = qb.invert_batched(A)
    assert list(info[[0, 1, 2, 3, 5]]) == [0] * 5 and info[4] == N // 2 + 1
    for b in (0, 1, 5):
        ref = np.linalg.inv(A[b])
        assert np.max(np.abs(inv[b] - ref)) < 1e-12 * np.max(np.abs(ref))
    if N <= 120:  # the kernels above scale no reciprocal (|a|^2 of a pivot has to be in range)
        ref = np.linalg.inv(well)
        assert np.max(np.abs(inv[2] * 1e250 - ref)) < 1e-12 * np.max(np.abs(ref))
        assert np.max(np.abs(inv[3] * 1e-250 - ref)) < 1e-12 * np.max(np.abs(ref))
