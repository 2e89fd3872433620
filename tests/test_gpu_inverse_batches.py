"""The batched inversion where a block does several matrices one after the other and where its kernels keep the
matrix in global memory: what one matrix leaves behind (a zero pivot, the places of its columns) must not reach the
next one, pivots may lie anywhere, and reciprocals are scaled. Tolerances as in test_gpu_inverse_orders.py."""
import numpy as np
import pytest

import quichotte_b200 as qb

pytestmark = pytest.mark.gpu


# more matrices than resident blocks: 592 up to order 96, 444 to 128, 296 above
@pytest.mark.parametrize("N, batch", [(33, 2500), (81, 1300), (96, 1300), (97, 900), (113, 900), (120, 900), (121, 900), (128, 700),
                                      (129, 620), (192, 620), (256, 320), (257, 310)])
def test_matrices_of_a_block_do_not_meet(N, batch):
    rng = np.random.default_rng(3 * N)
    eye = 3 * np.sqrt(N) * np.eye(N)
    noise = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    well = eye + 0.1 * noise
    singular = well.copy()
    singular[:, N // 2] = 0.0  # step N/2 + 1 finds no pivot
    kinds = [well, eye[::-1] + 0.01 * noise, singular, well * 1e250, well * 1e-250, noise + eye[rng.permutation(N)], eye * 1j]
    A = np.array([kinds[b % 7] for b in range(batch)])
    inv, info = qb.invert_batched(A)
    assert all(info[b] == (N // 2 + 1 if b % 7 == 2 else 0) for b in range(batch))
    for q in (0, 1, 3, 4, 5, 6):
        scale = {3: 1e250, 4: 1e-250}.get(q, 1.0)
        ref = np.linalg.inv(well if q in (3, 4) else kinds[q])
        assert np.max(np.abs(inv[q] * scale - ref)) < 1e-12 * np.max(np.abs(ref)), q
        assert all(np.array_equal(inv[b], inv[q]) for b in range(q, batch, 7)), q
