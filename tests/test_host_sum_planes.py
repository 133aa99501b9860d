"""mdg_gemm_host on blocks over sum planes (row panels of A by column strips of
B, k from 449 on): the bits of one device-side GEMM over digit pairs.  The
second panel and the last strip hold digits whose sums need flush groups of 4
k-steps and the rest does not, so a block that took the norm of another panel
or strip would be inexact."""
from fractions import Fraction

import numpy as np
import pytest

from conftest import pkg

# one strip, two panels; two strips, two panels; two strips, four panels
SHAPES = [(4, 2600, 700, 520), (2, 2304, 4300, 1030), (4, 4200, 4100, 600)]


def _entry(p, digits):
    """The entry whose balanced base-256 digits are `digits`."""
    v, limbs = sum(Fraction(d, 256 ** i) for i, d in enumerate(digits)) / 128, []
    for _ in range(p):
        limbs.append(float(v))
        v -= Fraction(limbs[-1])
    return np.array(limbs)


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,k", SHAPES)
def test_host_blocks_over_sum_planes(p, m, n, k):
    import torch
    api = pkg("api")
    digits = [-70] + [-127 if i & 1 else -128 for i in range(1, api.default_slices(p))]
    entry = torch.from_numpy(_entry(p, digits)).cuda()
    A = api.generate("normal", p, m, k, 41, -9, 9, scale_rows=True)
    B = api.generate("uniform", p, k, n, 42)
    panel = -(-(m // min(4, m // 1024)) // 256) * 256
    A[panel:panel + 300] = entry
    B[:, n - 250:] = entry
    want = api.gemm(A, B, engine="tc").cpu().numpy()
    hA, hB = A.cpu().numpy(), B.cpu().numpy()
    for _ in range(2):
        assert np.array_equal(api.gemm_host(hA, hB), want)
    assert api.device_status() == 0
