"""The renormalisation kernel (csrc/renorm.cuh) where its widths change: the
diagonal counts around whole 64-bit words, the two-column variant of large
outputs, diagonals of three and more chunks.  Against the oracle, bit for
bit."""
import numpy as np
import pytest

from conftest import pkg


def _check(orc, p, D, k, m, n, seed):
    import torch
    api = pkg("api")
    rng = np.random.default_rng(seed)
    nch = pkg("_lib").lib().mdg_slice_chunk_count(D, D, k)
    Cd = rng.integers(-(2 ** 31), 2 ** 31, size=(nch, m, n)).astype(np.int32)
    Cd[:, 0, : n // 2] = -1
    Cd[:, 1, :] = rng.integers(-1, 2, size=(nch, n)).astype(np.int32)
    Cd[1:, 2, :] = 0
    E = rng.integers(-60, 60, size=m).astype(np.int32)
    F = rng.integers(-60, 60, size=n).astype(np.int32)
    dCd = torch.from_numpy(Cd).cuda()
    got = api.renorm_diagonals(dCd, torch.from_numpy(E).cuda(), torch.from_numpy(F).cuda(), p, D,
                               D, k).cpu().numpy()
    diag = api.chunks_to_diagonals(dCd, D, D, k)
    assert np.array_equal(got, orc.renorm_diags(p, D, diag, E, F, m, n))


@pytest.mark.gpu
@pytest.mark.parametrize("p,D", [(2, 1), (4, 2), (2, 8), (4, 9), (8, 31), (4, 32), (8, 33),
                                 (16, 64), (16, 112)])
@pytest.mark.parametrize("k", [64, 300000])
def test_renorm_word_edges(orc, p, D, k):
    _check(orc, p, D, k, 7, 23, 100 * p + D)


@pytest.mark.gpu
@pytest.mark.parametrize("p,D,m,n,k", [(2, 14, 1024, 514, 64), (4, 28, 1030, 510, 20000),
                                       (8, 55, 524, 1002, 64)])
def test_renorm_two_columns(orc, p, D, m, n, k):
    _check(orc, p, D, k, m, n, D)


@pytest.mark.gpu
@pytest.mark.parametrize("p,D,m,n,k", [(4, 28, 256, 512, 5000), (4, 28, 255, 514, 5000),
                                       (2, 14, 361, 364, 64), (8, 55, 257, 511, 300)])
def test_renorm_where_two_columns_begin(orc, p, D, m, n, k):
    """Around 2^17 entries, odd rows of planes among them."""
    _check(orc, p, D, k, m, n, D + 1)
