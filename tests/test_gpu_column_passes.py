"""How many right-hand sides a solve takes in one pass over the factors: FP32 blocks 93..96 wide fit the
staged sweeps with a few columns only, and take the unstaged or streamed ones when there are more."""
import numpy as np
import pytest
import torch

import blockstructuredsolvers_gb300 as bss
from blockstructuredsolvers_gb300 import _lib
from oracle import cref
from oracle import oracle as O
from tests.gpu_util import download_x, upload

pytestmark = pytest.mark.gpu


def _launches(n, k, T, precision):
    """Kernel launches of one unrefined solve; its solution within the FP32 bound of the suite, 1e-4."""
    A, B, d = O.gen_shifted_family(np.random.default_rng(n), 61, n, k, diag_shift=2.0 * n, b_scale=0.5)
    data = bss.initialize_batched(61, n, T, k=k, precision=precision, max_refine=0, tol=1e-3, use_graphs=False)
    upload(data, A, B, d)
    bss.factorize_(data)
    before = _lib.load().bss_kernel_launches()
    bss.solve_(data)
    after = _lib.load().bss_kernel_launches()
    bss.synchronize(data)
    assert O.rel_error(download_x(data, 61), cref.solve_math(A, B, d, np.float64)) <= 1e-4
    return after - before


@pytest.mark.parametrize("T,precision", [(torch.float32, "plain"), (torch.float64, "mixed")])
@pytest.mark.parametrize("n,k,most", [(92, 8, 1.2), (93, 8, 1.2), (95, 16, 1.2), (96, 8, 2), (96, 16, 4)])
def test_passes(n, k, most, T, precision):
    """`most`: times the launches of one right-hand side's pass (its residual may take one more); the
    streamed sweeps (n = 96) have one more per level and take eight columns."""
    assert _launches(n, k, T, precision) <= most * _launches(n, 1, T, precision)
