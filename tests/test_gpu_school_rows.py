"""Thread-per-product schoolbook: every pair of lengths up to 16 limbs, batch
sizes around the CTA's 128 rows, strides, broadcast rows and all-ones
operands (every carry chain full).  Exact against Python integers."""
import numpy as np
import pytest

import batch_ref as ref
from helpers import rand_buf, to_dev

pytestmark = pytest.mark.gpu


def run(N, La, Lb, sA, sB, sC, ones, seed):
    import gpupi_b200 as g
    rng = np.random.default_rng(seed)
    A, B, C = rand_buf(rng, N, sA, La), rand_buf(rng, max(N if sB else 1, 1), sB or Lb, Lb), rand_buf(rng, N, sC, 0)
    if ones:
        A[:] = 0xFFFFFFFF
        B[:] = 0xFFFFFFFF
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C)
    g.mul_naive(N, dA.ptr, La, sA, dB.ptr, Lb, sB, dC.ptr, sC)
    assert np.array_equal(dC.numpy(), ref.mul(N, A, La, sA, B, Lb, sB, C, sC)), (N, La, Lb)


@pytest.mark.parametrize("La", range(1, 17))
def test_all_lengths(La):
    for Lb in range(1, 17):
        run(5, La, Lb, La, Lb, La + Lb, True, La * 16 + Lb)
        run(131, La, Lb, La, Lb, La + Lb, False, La * 17 + Lb)


@pytest.mark.parametrize("N", [1, 127, 128, 129, 1000])
def test_batches(N):
    run(N, 13, 14, 15, 14, 30, False, N)
    run(N, 16, 3, 16, 0, 19, False, N)
    run(N, 2, 16, 5, 16, 18, False, N)
