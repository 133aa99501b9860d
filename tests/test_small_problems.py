"""The BF16 form on problems of few tiles: chunks cut so that every CTA gets
a share, narrow tiles for up to 128 rows or columns, two diagonals in one
accumulator where that pads less.  The same bits from the
automatic choice, the CTA-pair, the single-CTA and the mma.sync engine."""
import pytest

from conftest import pkg


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,k", [
    (2, 1, 1, 1), (2, 64, 64, 64), (4, 128, 128, 65), (4, 129, 128, 300), (4, 128, 129, 1000),
    (4, 256, 256, 256), (4, 257, 500, 640), (8, 100, 1000, 130), (8, 1000, 100, 77),
    (16, 130, 130, 129), (2, 16001, 96, 100), (4, 96, 3000, 600), (2, 60, 60, 20000),
    (4, 512, 512, 200), (8, 700, 300, 900),
    # many tiles of 128 rows or columns: two diagonals per accumulator (even
    # and odd digit counts, k ending inside a block)
    (2, 100, 33000, 130), (2, 20000, 300, 70), (8, 20000, 100, 40), (8, 128, 25000, 33),
    (4, 9000, 384, 200)])
def test_few_tiles_same_bits(p, m, n, k):
    import torch
    api = pkg("api")
    A = api.generate("normal", p, m, k, 7, -9, 9, scale_rows=True)
    B = api.generate("uniform", p, k, n, 8)
    got = api.gemm(A, B)
    for engine in ("tc", "tc_pair", "mma_sync"):
        assert torch.equal(got, api.gemm(A, B, engine=engine)), engine
    assert torch.equal(got, api.gemm(A, B, parts=3))
    assert api.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("p,m,n,k", [
    # digit pairs over a few tiles, a run of diagonals a unit: stacked on either
    # side (odd and even digit counts), unstacked, as many units as fit the
    # argument (2, 37000, 64: 145 x 7 = 1015) and one tile row more (1022), one
    # more again (1029: in turn)
    (8, 3000, 64, 100), (16, 100, 1000, 90), (4, 2000, 300, 450), (2, 900, 900, 300),
    (16, 500, 500, 70), (2, 37000, 64, 70), (2, 37200, 100, 40), (2, 37500, 64, 40)])
def test_dealt_units_same_bits(p, m, n, k):
    import torch
    api = pkg("api")
    A = api.generate("uniform", p, m, k, 17, -9, 9, scale_rows=True)
    B = api.generate("normal", p, k, n, 18)
    got = api.gemm(A, B)
    assert torch.equal(got, api.gemm(A, B, parts=1))
    assert torch.equal(got, api.gemm(A, B, engine="tc"))
    assert api.device_status() == 0
