"""FP64 chain kernels with digit products on the tensor cores
(csrc/bss_chain_f64_tc.cuh, csrc/bss_chain128_f64_tc.cuh): all tile sizes and their remainders, chains with
and without separators, rows of very different sizes, and non-finite blocks."""
import numpy as np
import pytest
import torch

import blockstructuredsolvers_gb300 as bss
from oracle import cref
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _handle(A, B, d, parts):
    N, n, k = d.shape
    if parts == 0:
        data = bss.initialize_seq(N, n, torch.float64, k=k)
    else:
        data = bss.initialize_batched(N, n, torch.float64, k=k, target_partitions=parts)
    data.A_tensor[:, :, :N] = torch.from_numpy(A).cuda().permute(1, 2, 0)
    data.B_tensor[:, :, :N - 1] = torch.from_numpy(B).cuda().permute(1, 2, 0)
    data.d_tensor[:, :, :N] = torch.from_numpy(d).cuda().permute(1, 2, 0)
    return data


def _solve(data, N):
    bss.factorize_(data)
    bss.solve_(data)
    bss.synchronize(data)
    return data.d_tensor[:, :, :N].permute(2, 0, 1).cpu().numpy()


@pytest.mark.parametrize("parts", [0, 1, 3])
@pytest.mark.parametrize("n", [17, 24, 31, 32, 33, 40, 49, 63, 64, 65, 72, 97, 127, 128])
def test_against_oracle(n, parts):
    rng = np.random.default_rng(100 * n + parts)
    A, B, d = O.gen_shifted_family(rng, 17, n, 2, diag_shift=2.0 * n, b_scale=0.5)
    x = _solve(_handle(A, B, d, parts), 17)
    assert O.rel_error(x, cref.solve_math(A, B, d, np.float64)) <= 1e-10


@pytest.mark.parametrize("n", [32, 37, 64, 70, 128])
def test_rows_of_different_sizes(n):
    """T -> D T D with D = diag(2^-12 .. 2^12): digits are cut row by row, so every
    row keeps its own precision.  Backward error of a block Cholesky is a small
    multiple of n u (n = 128: 1.4e-14): 1e-13 with the widened row norms."""
    rng = np.random.default_rng(n)
    A, B, d = O.gen_shifted_family(rng, 19, n, 1, diag_shift=2.0 * n, b_scale=0.5)
    D = 2.0 ** rng.integers(-12, 13, (19, n))
    A = D[:, :, None] * A * D[:, None, :]
    B = D[:-1, :, None] * B * D[1:, None, :]
    d = D[:, :, None] * d
    x = _solve(_handle(A, B, d, 2), 19)
    assert O.rel_residual(A, B, x, d) <= 1e-13


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["A", "B"])
@pytest.mark.parametrize("n", [32, 64, 100])
def test_non_finite_blocks_are_reported(n, where, value):
    rng = np.random.default_rng(n)
    A, B, d = O.gen_shifted_family(rng, 11, n, 1, diag_shift=2.0 * n, b_scale=0.5)
    if where == "A":
        A[4, 3, 3] = value
    else:
        B[4, 2, 5] = value
    data = _handle(A, B, d, 0)
    with pytest.raises(bss.NotSPDError):
        _solve(data, 11)
