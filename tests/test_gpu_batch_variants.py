"""Batches take the factor kernel that their handles' variant names (bss_diag_set_factor_variant before the
batch is created), as single systems do: the CUDA-core chain kernel for 33..64-wide blocks, the L2-staged
wide kernel for 65..128.  The two kernels round differently, so the variant shows in the bits."""
import numpy as np
import pytest
import torch

import blockstructuredsolvers_gb300 as bss
from blockstructuredsolvers_gb300 import _lib
from oracle import cref
from oracle import oracle as O
from tests.gpu_util import download_x, upload

pytestmark = pytest.mark.gpu


def _batch(probs, shapes, variant):
    L = _lib.load()
    saved = L.bss_diag_get_factor_variant()
    _lib.check(L.bss_diag_set_factor_variant(variant))
    try:
        b = bss.initialize_multi(*(list(s) for s in zip(*shapes)), torch.float32)
    finally:
        _lib.check(L.bss_diag_set_factor_variant(saved))
    for s, p in zip(b.systems, probs):
        upload(s, *p)
    b.factorize()
    b.solve()
    b.synchronize()
    return [download_x(s, s.N) for s in b.systems]


@pytest.mark.parametrize("variant,n", [(1, 40), (1, 64), (2, 70), (2, 128)])
def test_variant_reaches_the_batch(variant, n):
    """FP32 solutions against the FP64 oracle at the suite's 1e-4."""
    shapes = [(300, n, 1), (261, n, 2), (280, 24, 1)]  # the last has one kernel whatever the variant
    probs = [O.gen_shifted_family(np.random.default_rng(n + i), *s, diag_shift=2.0 * s[1], b_scale=0.5)
             for i, s in enumerate(shapes)]
    refs = [cref.solve_math(*p, np.float64) for p in probs]
    default, chosen = _batch(probs, shapes, 0), _batch(probs, shapes, variant)
    for x, y, ref in zip(default, chosen, refs):
        assert O.rel_error(x, ref) <= 1e-4 and O.rel_error(y, ref) <= 1e-4
    for x, y in zip(default[:2], chosen[:2]):
        assert not np.array_equal(x, y)
    assert np.array_equal(default[2], chosen[2])
