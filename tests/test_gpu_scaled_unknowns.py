"""Plain FP64 systems whose unknowns have different units: T -> D T D with D a power of two of its
own for every unknown.  Every FP64 product, sum, reciprocal and square root of the factorization and
the solve is homogeneous in such a D, so D times the scaled system's solution is the unscaled one,
with the unscaled solution's error; the normwise residual of the scaled system cannot show a loss
(its norms are inflated by D), so the solutions are compared."""
import numpy as np
import pytest
import torch

import blockstructuredsolvers_gb300 as bss
from oracle import cref
from oracle import oracle as O
from tests.gpu_util import download_x, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [12, 27, 40])
@pytest.mark.parametrize("parts", [0, 1, 3])
@pytest.mark.parametrize("n", [16, 17, 32, 37, 64, 65, 70, 128])
def test_solution_does_not_depend_on_units(n, parts, spread):
    """Tolerance: a few n u for this well-conditioned family (128 u = 1.4e-14), 1e-12 with room for
    the chain's length and the condition number."""
    rng = np.random.default_rng(1000 * n + 10 * parts + spread)
    N = 19
    A, B, d = O.gen_shifted_family(rng, N, n, 1, diag_shift=2.0 * n, b_scale=0.5)
    x_ref = cref.solve_math(A, B, d, np.float64)
    D = 2.0 ** rng.integers(-spread, spread + 1, (N, n))
    if parts == 0:
        data = bss.initialize_seq(N, n, torch.float64)
    else:
        data = bss.initialize_batched(N, n, torch.float64, target_partitions=parts)
    upload(data, D[:, :, None] * A * D[:, None, :], D[:-1, :, None] * B * D[1:, None, :], D[:, :, None] * d)
    bss.factorize_(data)
    bss.solve_(data)
    bss.synchronize(data)
    assert O.rel_error(D[:, :, None] * download_x(data, N), x_ref) <= 1e-12
