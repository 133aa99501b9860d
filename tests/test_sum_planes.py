"""The diagonal sums from products of sum planes (csrc/cross_sums.cuh), the
route of large BF16-form problems: the same bits as the digit pairs (the
single-CTA engine, itself checked against the oracle) on ragged shapes, at
every limb count, with digits that force each flush interval, and in a
workspace that only holds the pairs."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from conftest import pkg


def test_workspace_holds_the_pairs_and_the_rule_is_on_sizes():
    api, L = pkg("api"), pkg("_lib").lib()
    for p, m, n, k, sums in [(4, 1024, 1024, 1024, True), (2, 16001, 96, 3001, False),
                             (4, 4096, 4096, 256, False), (8, 2048, 2048, 2048, True), (16, 1024, 1024, 512, True),
                             (4, 1024, 1024, 70000, False), (4, 65536, 65536, 8192, False)]:
        full = api.workspace_size("slice_bf16", p, m, n, k)
        least = L.mdg_gemm_least_workspace_size(2, p, m, n, k, None)
        assert (full > least) if sums else (full == least), (p, m, n, k)
    assert L.mdg_gemm_least_workspace_size(0, 4, 8, 8, 8, None) == 0
    assert L.mdg_gemm_least_workspace_size(2, 3, 8, 8, 8, None) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,k,kw", [
    (4, 1024, 1024, 512, {}),             # the least k: groups of 8 k-steps
    (4, 1000, 777, 1031, {}),             # k-steps that 16 does not divide, ragged tiles
    (4, 257, 300, 1025, {}),              # four tiles, most of them padding
    (2, 1100, 1030, 1024, {}),
    (8, 1023, 800, 1100, {}),
    (16, 800, 1024, 1024, {}),
    (4, 300, 200, 40000, {}),             # one pair a chunk
    (4, 500, 400, 9000, {"parts": 5}),    # several pairs a chunk, several chunks a diagonal
    (4, 1024, 1024, 1024, {"diagonals": 21}),
    (4, 1024, 1024, 1024, {"slices": 30, "diagonals": 29, "engine": "tc_pair"}),
])
def test_sum_planes_give_the_bits_of_the_digit_pairs(p, m, n, k, kw):
    import torch
    api = pkg("api")
    A = api.generate("normal", p, m, k, 5, -20, 20, scale_rows=True)
    B = api.generate("uniform", p, k, n, 6)
    ref = dict(kw, engine="tc")
    ref.pop("parts", None)
    assert torch.equal(api.gemm(A, B, **kw), api.gemm(A, B, **ref))
    assert api.device_status() == 0


def _constant(api, p, rows, cols, digits):
    """rows x cols equal entries whose balanced digits are `digits`."""
    v, limbs = sum(Fraction(d, 256 ** i) for i, d in enumerate(digits)) / 128, []
    for _ in range(p):
        limbs.append(float(v))
        v -= Fraction(limbs[-1])
    return np.tile(np.array(limbs), (rows, cols, 1))


@pytest.mark.gpu
@pytest.mark.parametrize("even,odd", [(-20, -21), (-70, -71), (-128, -127)])
def test_flush_interval_follows_the_digits(even, odd):
    """Sums of equal sign and odd value in every product: 1024 products of
    41^2 stay below 2^24, of 141^2 only 512 do, of 255^2 only 256."""
    import torch
    api = pkg("api")
    p, n = 4, 1024
    digits = [-70] + [odd if i & 1 else even for i in range(1, api.default_slices(p))]
    X = torch.from_numpy(_constant(api, p, n, n, digits)).cuda()
    X[::3] *= -1
    E, F = api.scale_exponents(X, X)
    got = api.slice_digits(X, E, len(digits))[:, 1, 0].cpu().float().tolist()
    assert got[1:len(digits) - 8] == [float(d) for d in digits[1:len(digits) - 8]]
    assert torch.equal(api.gemm(X, X), api.gemm(X, X, engine="tc"))


@pytest.mark.gpu
def test_smaller_workspace_gives_the_same_bits():
    import torch
    api, L = pkg("api"), pkg("_lib").lib()
    p, n = 4, 1024
    A, B = api.generate("uniform", p, n, n, 1), api.generate("uniform", p, n, n, 2)
    ref, C = api.gemm(A, B), torch.empty_like(A)
    least = L.mdg_gemm_least_workspace_size(2, p, n, n, n, None)
    ws = torch.empty(least, dtype=torch.uint8, device="cuda")
    args = (2, p, n, n, n, A.data_ptr(), n, B.data_ptr(), n, C.data_ptr(), n, None, ws.data_ptr())
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.mdg_gemm(*args, least, st) == 0
    assert torch.equal(C, ref)
    assert L.mdg_gemm(*args, least - 1, st) == 5


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,k", [
    # units dealt to the clusters: more clusters than tiles, chunks of several
    # planes and of one, tiles at the argument's limit; the last beyond the
    # sizes that are dealt
    (4, 1000, 777, 1531), (16, 900, 1000, 530), (2, 1500, 1300, 16000), (2, 3000, 3000, 1024),
    (8, 1500, 1500, 1100)])
def test_dealt_sums_same_bits(p, m, n, k):
    import torch
    api = pkg("api")
    A = api.generate("normal", p, m, k, 21, -9, 9, scale_rows=True)
    B = api.generate("uniform", p, k, n, 22)
    got = api.gemm(A, B)
    assert torch.equal(got, api.gemm(A, B, parts=1))
    assert torch.equal(got, api.gemm(A, B, engine="tc"))
    assert api.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,k,kw", [
    # the renormalisation without prefix sums: 33 diagonals and more, one chunk a
    # diagonal; one and two columns a thread, odd columns; the k from which the
    # longest diagonals have two chunks (28 pairs of 36 and 37 k-blocks)
    (4, 1000, 777, 1024, {"slices": 33, "diagonals": 33}),
    (8, 600, 611, 1024, {}), (8, 800, 777, 64 * 36, {}), (8, 800, 777, 64 * 37, {}),
    (16, 600, 700, 700, {}), (16, 800, 801, 513, {})])
def test_renorm_of_whole_diagonals(p, m, n, k, kw):
    import torch
    api = pkg("api")
    A = api.generate("normal", p, m, k, 31, -9, 9, scale_rows=True)
    B = api.generate("uniform", p, k, n, 32)
    assert torch.equal(api.gemm(A, B, **kw), api.gemm(A, B, engine="tc", **kw))


@pytest.mark.gpu
@pytest.mark.parametrize("even,odd,infinite", [(-70, -71, False), (-128, -127, False),
                                               (-128, -127, True)])
def test_flush_interval_of_uneven_digits(even, odd, infinite):
    """Products of sums of about 141^2 and 255^2 that differ from k to k, so that
    1024 of them lose bits in FP32.  infinite: besides, a row of A and a column of
    B with an infinity and digits beyond 128; the norms of their sums, 2^31 each,
    must not make the interval of the others longer (4 x 2^62 is 0 modulo 2^64)."""
    import torch
    api = pkg("api")
    p, n, r, c = 4, 1024, 5, 7
    digits = [-70] + [odd if i & 1 else even for i in range(1, api.default_slices(p))]
    one, two = (torch.from_numpy(_constant(api, p, n, n, x)).cuda()
                for x in (digits, [d + (i & 1) for i, d in enumerate(digits)]))
    g = torch.Generator(device="cuda").manual_seed(1)
    A, B = (torch.where(torch.rand((n, n, 1), generator=g, device="cuda") < 0.5, one, two)
            for _ in range(2))
    if infinite:
        A[r] = 0
        A[r, 0, 0] = float("inf")
        e = int(api.scale_exponents(A, B)[0][r])
        A[r, 1:3, 0] = 2.0 ** (8 + e)  # leading digit 2^15, twice in a window
        B[:, c] = A[r]
        d = api.slice_digits(A, api.scale_exponents(A, B)[0], len(digits))[:, r].float()
        assert d[0, 1:3].tolist() == [2.0 ** 15] * 2 and float(d.abs().sum()) == 2.0 ** 16
    got, want = api.gemm(A, B), api.gemm(A, B, engine="tc")
    if infinite:
        for x in (got, want):
            x[r] = 0
            x[:, c] = 0
    assert torch.equal(got, want)


@pytest.mark.gpu
@pytest.mark.parametrize("digits", [47, 48, 49])
def test_digit_rows_around_the_default_shared_memory_limit(digits):
    """48 digit rows of 1 KiB and a few bytes of static memory are more than a
    block gets unasked."""
    import torch
    api = pkg("api")
    A, B = api.generate("uniform", 4, 800, 1024, 61), api.generate("normal", 4, 1024, 800, 62)
    kw = {"slices": digits, "diagonals": digits}
    assert torch.equal(api.gemm(A, B, **kw), api.gemm(A, B, engine="tc", **kw))
