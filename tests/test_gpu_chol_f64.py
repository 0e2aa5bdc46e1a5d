"""FP64 Cholesky + inverse of the chain kernels' pivot blocks
(csrc/bss_chol_f64.cuh): every panel count and remainder of the tile sizes,
and pivots whose exponents leave the range of the FP32-seeded reciprocal,
against the C oracle."""
import numpy as np
import pytest
import torch

import blockstructuredsolvers_gb300 as bss
from oracle import cref
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _solve(A, B, d):
    N, n, k = d.shape
    data = bss.initialize_batched(N, n, torch.float64, k=k)
    data.A_tensor[:, :, :N] = torch.from_numpy(A).cuda().permute(1, 2, 0)
    data.B_tensor[:, :, :N - 1] = torch.from_numpy(B).cuda().permute(1, 2, 0)
    data.d_tensor[:, :, :N] = torch.from_numpy(d).cuda().permute(1, 2, 0)
    bss.factorize_(data)
    bss.solve_(data)
    bss.synchronize(data)
    return data.d_tensor[:, :, :N].permute(2, 0, 1).cpu().numpy()


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64, 80, 128])
@pytest.mark.parametrize("exponent", [0, -1000, 1000])
def test_pivot_blocks(n, exponent):
    """A and B scaled by 2^exponent (exact): x scales by 2^-exponent exactly, so the
    unscaled oracle solution stands for all three.  d is scaled with them where the
    solution would leave the FP64 range.  Tolerance: the suite's FP64 bound 1e-10."""
    rng = np.random.default_rng(n)
    A, B, d = O.gen_shifted_family(rng, 13, n, 2, diag_shift=2.0 * n, b_scale=0.5)
    x_ref = cref.solve_math(A, B, d, np.float64)
    s = 2.0 ** exponent
    x = _solve(A * s, B * s, d * s)
    assert O.rel_error(x, x_ref) <= 1e-10
