"""Forms of the chain kernels and solve sweeps at the sizes where they change:
the kernel for blocks up to 16 wide, sweeps over few and many partitions (whose
coarser levels form their right-hand side themselves and start under the level
before) for every column form, and the batch's queue forms.  Each is solved
twice (the first call launches, the second replays a graph).

Tolerances, as everywhere in this suite for these well-conditioned families:
relative error against the block Cholesky in FP64 <= 1e-10 (FP64 and mixed) or
<= 1e-4 (FP32), relative residual <= 1e-12 (mixed)."""
import numpy as np
import pytest
import torch

import blockstructuredsolvers_gb300 as bss
from oracle import cref
from oracle import oracle as O
from tests.gpu_util import download_x, upload

pytestmark = pytest.mark.gpu

KINDS = {"f32": (torch.float32, "plain"), "f64": (torch.float64, "plain"), "mixed": (torch.float64, "mixed")}


def _gen(seed, N, n, k):
    return O.gen_shifted_family(np.random.default_rng(seed), N, n, k, diag_shift=2.0 * max(n, 6), b_scale=0.5)


def _check(kind, A, B, d, x, x_ref):
    assert O.rel_error(x, x_ref) <= (1e-4 if kind == "f32" else 1e-10)
    if kind == "mixed":
        assert O.rel_residual(A, B, x, d) <= 1e-12


def _run(kind, N, n, k, parts):
    A, B, d = _gen(1000 * n + 10 * k + parts, N, n, k)
    T, precision = KINDS[kind]
    if parts == 0:
        data = bss.initialize_seq(N, n, T, k=k)
    else:
        data = bss.initialize_batched(N, n, T, k=k, precision=precision, target_partitions=parts)
    x_ref = cref.solve_math(A, B, d, np.float64)
    for _ in range(2):
        upload(data, A, B, d)
        bss.factorize_(data)
        bss.solve_(data)
        bss.synchronize(data)
        _check(kind, A, B, d, download_x(data, N), x_ref)


@pytest.mark.parametrize("parts", [0, 1, 5])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_blocks_up_to_16(kind, n, parts):
    if kind == "mixed" and parts == 0:
        pytest.skip("the sequential form has no mixed precision")
    _run(kind, 23, n, 2, parts)


@pytest.mark.parametrize("n,k", [(3, 1), (16, 16), (24, 2), (32, 3), (37, 4), (48, 5), (63, 1), (64, 16), (65, 1),
                                 (96, 2), (112, 9), (127, 3), (128, 1), (128, 8)])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_sweeps_of_many_levels(kind, n, k):
    _run(kind, 83, n, k, 20)


@pytest.mark.parametrize("n,k", [(8, 1), (16, 4), (32, 1)])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_more_partitions_than_two_per_sm(kind, n, k):
    _run(kind, 1300, n, k, 400)


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_batch_queue_forms(kind):
    T, precision = KINDS[kind]
    wide_k = 9 if kind == "f32" else 2  # a batch takes what fits one solve pass
    systems = [(1, 128, 1), (2, 65, 2), (40, 33, 1), (70, 47, 3), (66, 64, 16 if kind == "f32" else 4), (41, 66, 1),
               (70, 100, 8 if kind == "f32" else 2), (35, 112, wide_k), (90, 128, 2), (50, 16, 1), (45, 9, 5),
               (130, 32, 2)]
    probs = [_gen(7 + i, *s) for i, s in enumerate(systems)]
    refs = [cref.solve_math(*p, np.float64) for p in probs]
    b = bss.initialize_multi([s[0] for s in systems], [s[1] for s in systems], [s[2] for s in systems], T,
                             precision=precision)
    for _ in range(2):
        for s, p in zip(b.systems, probs):
            upload(s, *p)
        b.factorize()
        b.solve()
        b.synchronize()
        for s, (A, B, d), x_ref in zip(b.systems, probs, refs):
            _check(kind, A, B, d, download_x(s, s.N), x_ref)
