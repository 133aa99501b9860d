"""The device's three-operation two-sum (include/mdg_arith.h) where it has a
case of its own: operands in either order, errors of -0, sums of opposite
zeros, subnormals, sums that overflow.  Through the plain form with k = 2 and
3, against the oracle, which has the six operations: the same values, the same
signs of zero and NaN in the same places."""
import numpy as np
import pytest

from conftest import pkg


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 4, 8])
@pytest.mark.parametrize("k", [2, 3])
def test_two_sum_cases(orc, p, k):
    import torch
    api = pkg("api")
    hi = np.array([0.0, -0.0, 1.0, -1.0, 1.0 + 2.0 ** -52, -(1.0 - 2.0 ** -53), 3.0 * 2.0 ** 52,
                   2.0 ** -1074, -2.0 ** -1022, 1.5 * 2.0 ** 1023, -1.5 * 2.0 ** 1023])
    rng = np.random.default_rng(10 * p + k)
    m = n = 44
    A = np.zeros((m, k, p))
    B = np.zeros((k, n, p))
    A[..., 0] = rng.choice(hi, size=(m, k))
    B[..., 0] = rng.choice(np.array([1.0, -1.0, 0.0, -0.0]), size=(k, n))
    A[..., 1] = rng.choice(np.array([0.0, -0.0, 2.0 ** -60, -2.0 ** -60]), size=(m, k))
    A[..., 1][np.abs(A[..., 0]) < 0.5] = -0.0
    got = api.gemm(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), "plain").cpu().numpy()
    want = orc.gemm_plain(p, A, B, m, n, k)
    assert np.array_equal(got, want, equal_nan=True)
    fin = ~np.isnan(want)
    assert np.array_equal(np.signbit(got[fin]), np.signbit(want[fin]))
