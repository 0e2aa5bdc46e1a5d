"""Right-hand sides near the end of the FP32 range: a separator's right-hand side minus its two neighbours'
contributions stays in range although the first difference alone does not."""
import numpy as np
import pytest
import torch

import blockstructuredsolvers_gb300 as bss
from oracle import cref
from oracle import oracle as O
from tests.gpu_util import download_x, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8])
def test_separator_rhs_near_overflow(n):
    """Separators at the even blocks; d is 2.5e38 at block 8 and its left neighbour, -2.5e38 at the right one,
    and the couplings are 0.49 of the diagonal, so d_8 - bL is 3.7e38 (beyond FP32) and d_8 - bL - bR 2.5e38.
    FP32 tolerance of the suite: 1e-4."""
    N = bss.initialize_batched(21, n, torch.float32).A_tensor.shape[2]  # blocks of the padded system
    assert N % 2 == 1
    A = np.tile(100.0 * np.eye(n), (21, 1, 1))
    B = np.tile(49.0 * np.eye(n), (20, 1, 1))
    d = np.zeros((21, n, 1))
    d[7], d[8], d[9] = 2.5e38, 2.5e38, -2.5e38
    data = bss.initialize_batched(21, n, torch.float32, target_partitions=(N - 1) // 2)
    upload(data, A, B, d)
    bss.factorize_(data)
    bss.solve_(data)
    bss.synchronize(data)
    assert O.rel_error(download_x(data, 21) / 1e38, cref.solve_math(A, B, d / 1e38, np.float64)) <= 1e-4
