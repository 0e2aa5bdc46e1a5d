"""Transpose products of the solve sweeps at the block sizes and right-hand sides where their form or their
walk through shared memory changes: chunks of 16, 8 and 4 bytes with every turn, and the FP64 form of whole
outputs per thread (blocks of up to four columns, half-empty tiles, threads whose four right-hand sides fill)."""
import numpy as np
import pytest
import torch

import blockstructuredsolvers_gb300 as bss
from oracle import cref
from oracle import oracle as O
from tests.gpu_util import download_x, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [0, 9])
@pytest.mark.parametrize("n,k", [(2, 12), (2, 32), (4, 11), (4, 12), (4, 32), (10, 24), (10, 25), (26, 32), (42, 24), (58, 16),
                                 (12, 1), (28, 1), (30, 3), (37, 1), (45, 2), (54, 5), (60, 16), (62, 2), (91, 1), (92, 3),
                                 (94, 2)])
@pytest.mark.parametrize("T", [torch.float64, torch.float32])
def test_against_oracle(T, n, k, parts):
    """The suite's bounds for this family: 1e-10 (FP64), 1e-4 (FP32)."""
    A, B, d = O.gen_shifted_family(np.random.default_rng(100 * n + k), 40, n, k, diag_shift=2.0 * max(n, 6), b_scale=0.5)
    data = bss.initialize_seq(40, n, T, k=k) if parts == 0 else bss.initialize_batched(40, n, T, k=k, target_partitions=parts)
    upload(data, A, B, d)
    bss.factorize_(data)
    bss.solve_(data)
    bss.synchronize(data)
    assert O.rel_error(download_x(data, 40), cref.solve_math(A, B, d, np.float64)) <= (1e-10 if T == torch.float64 else 1e-4)
