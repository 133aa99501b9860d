"""The digit and scale kernels (csrc/slice_stages.cuh) where they can go
wrong: digit counts around whole 32-bit pieces, odd widths (one k-position a
thread), operands off 16-byte alignment, few rows of great depth (ranges of
k), limbs of any order and exponent, NaN.  Digits against the
oracle, bit for bit; scale exponents against numpy."""
import numpy as np
import pytest

from conftest import pkg


def _cuda(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _limbs(rng, rows, cols, p):
    """Limbs of every magnitude in no order, zeros among them."""
    x = np.ldexp(rng.uniform(-1, 1, (rows, cols, p)), rng.integers(-900, 8, (rows, cols, p)))
    x[rng.random(x.shape) < 0.1] = 0.0
    x[rng.random(x.shape) < 0.05] = 5e-324
    return x


@pytest.mark.gpu
@pytest.mark.parametrize("p,s", [(2, 1), (2, 4), (4, 5), (2, 8), (4, 9), (8, 57), (16, 112)])
@pytest.mark.parametrize("cols", [1, 6, 131])
@pytest.mark.parametrize("trans", [False, True])
def test_digits_at_piece_edges(orc, p, s, cols, trans):
    api = pkg("api")
    rng = np.random.default_rng(100 * s + cols)
    rows = 5
    X = _limbs(rng, cols if trans else rows, rows if trans else cols, p)
    dX = _cuda(X)
    flip = dX.transpose(0, 1).contiguous()
    E = api.scale_exponents(flip, dX)[1] if trans else api.scale_exponents(dX, flip)[0]
    got = api.slice_digits(dX, E, s, trans=trans).float().cpu().numpy()
    want = orc.digits(p, s, X, rows, cols, E.cpu().numpy(), trans)
    assert np.array_equal(got, np.asarray(want, dtype=np.float32).reshape(got.shape))


@pytest.mark.gpu
def test_operands_off_16_byte_alignment():
    import torch
    api = pkg("api")
    for p, m, n, k in [(2, 40, 50, 70), (4, 33, 20, 65), (16, 20, 24, 30)]:
        A, B = api.generate("normal", p, m, k, 1), api.generate("uniform", p, k, n, 2)
        flat = torch.empty(A.numel() + 1, dtype=torch.float64, device="cuda")
        flat[1:] = A.reshape(-1)
        odd = flat[1:].view(m, k, p)
        assert odd.data_ptr() % 16 == 8 and odd.is_contiguous()
        C = torch.empty(m * n * p + 1, dtype=torch.float64, device="cuda")[1:].view(m, n, p)
        assert torch.equal(api.gemm(odd, B, out=C), api.gemm(A, B))


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(3, 2, 40000), (1, 700, 5000), (900, 9, 1025), (17, 33, 1)])
def test_scale_exponents_of_any_shape(m, n, k):
    api = pkg("api")
    rng = np.random.default_rng(k)
    A = np.ldexp(rng.uniform(-1, 1, (m, k, 2)), rng.integers(-300, 300, (m, k, 1)))
    B = np.ldexp(rng.uniform(-1, 1, (k, n, 2)), rng.integers(-300, 300, (k, n, 1)))
    A[0, 0] = [np.nan, 1.0]
    E, F = api.scale_exponents(_cuda(A), _cuda(B))
    for X, got, axis in ((A, E, 1), (B, F, 0)):
        v = np.abs(X[..., 0]) + np.abs(X[..., 1])
        M = np.nanmax(np.where(np.isnan(v), 0.0, v), axis=axis)
        frac, e = np.frexp(M)
        e = np.where(frac > 1 - 2.0 ** -29, e + 1, e)
        assert np.array_equal(got.cpu().numpy(), np.where(M > 0, e, 0))


@pytest.mark.gpu
def test_nan_entries_count_as_zero():
    """Their exponent lies far above the row's scale, so no digit of the
    row's range sees them."""
    import torch
    api = pkg("api")
    p, n = 4, 64
    A, B = api.generate("uniform", p, n, n, 1), api.generate("uniform", p, n, n, 2)
    Z = A.clone()
    Z[3, 5], Z[7, 1] = 0.0, 0.0
    A[3, 5], A[7, 1] = float("nan"), float("nan")
    assert torch.equal(api.gemm(A, B), api.gemm(Z, B))
