"""mdg_gemm_ex of the BF16 form, which reads transposed operands in place:
the bits of gemm on transposed copies, on the routes of large problems (sum
planes), few tiles and deep narrow ones (ranges of k), with padded rows."""
import pytest

from conftest import pkg


@pytest.mark.gpu
@pytest.mark.parametrize("ta,tb", [(False, True), (True, False), (True, True)])
@pytest.mark.parametrize("p,m,n,k", [(4, 1030, 1000, 1100), (2, 131, 70, 300), (8, 5, 9, 6000),
                                     (16, 64, 33, 50), (2, 4, 40000, 64)])
def test_transposed_operands_match_copies(p, m, n, k, ta, tb):
    import torch
    api = pkg("api")
    A, B = api.generate("normal", p, m, k, 3, -9, 9, scale_rows=True), api.generate("uniform", p, k, n, 4)
    ref = api.gemm(A, B)

    def stored(X, trans, pad):
        Y = X.transpose(0, 1).contiguous() if trans else X
        wide = torch.full((Y.shape[0], Y.shape[1] + pad, p), float("nan"), dtype=torch.float64,
                          device="cuda")
        wide[:, :Y.shape[1]] = Y
        return wide[:, :Y.shape[1]]

    got = api.gemm_ex(stored(A, ta, 3), stored(B, tb, 1), trans_a=ta, trans_b=tb)
    assert torch.equal(got, ref)
    C = api.generate("uniform", p, m, n, 5)
    want = api.gemm_ex(A, B, C=C.clone(), accumulate=True)
    assert torch.equal(api.gemm_ex(stored(A, ta, 0), stored(B, tb, 2), trans_a=ta, trans_b=tb,
                                   C=C, accumulate=True), want)


@pytest.mark.gpu
def test_workspace_between_the_least_and_the_fastest():
    """Short chunks of a small problem need more output planes; a workspace
    without room for them runs the plain chunks."""
    import ctypes
    import torch
    api, L = pkg("api"), pkg("_lib").lib()
    p, n = 4, 256
    full = L.mdg_gemm_workspace_size(2, p, n, n, n, None)
    least = L.mdg_gemm_least_workspace_size(2, p, n, n, n, None)
    assert least < full
    A, B = api.generate("uniform", p, n, n, 1), api.generate("uniform", p, n, n, 2)
    ref, C = api.gemm(A, B), torch.empty_like(A)
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for size in (least, (least + full) // 2, full):
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        C.zero_()
        assert L.mdg_gemm(2, p, n, n, n, A.data_ptr(), n, B.data_ptr(), n, C.data_ptr(), n, None,
                          ws.data_ptr(), size, st) == 0
        assert torch.equal(C, ref)
