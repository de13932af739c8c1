"""qdkp_block_gram of complex64 blocks that one CTA holds whole (split TF32): rows that end inside a chunk or
a part, leading dimensions with NaN beyond the columns, odd widths, and a block against itself. The entries are
small whole numbers, whose products and sums TF32 and FP32 hold exactly, so the results are exact."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize('n, P, Q, lda, ldb', [
    (1, 1, 1, 1, 1), (7, 3, 2, 3, 2), (7, 3, 2, 4, 3), (31, 12, 12, 12, 12), (33, 5, 24, 7, 24), (255, 18, 12, 19, 12),
    (256, 18, 12, 18, 12), (257, 18, 12, 18, 13), (1023, 13, 1, 13, 3), (1024, 36, 24, 36, 24), (1025, 36, 36, 37, 36),
    (4099, 39, 26, 41, 26), (4100, 39, 26, 40, 28), (75_777, 18, 12, 18, 12), (75_775, 48, 34, 48, 35),
    (151_553, 12, 5, 12, 5)])
def test_gram_of_complex64_blocks(n, P, Q, lda, ldb):
    import torch
    from qd3dsolver_b200 import _lib
    L = _lib.lib()
    g = torch.Generator('cuda').manual_seed(n + P)

    def block(cols, ld):
        a = torch.full((n, ld), float('nan'), dtype=torch.complex64, device='cuda')
        a[:, :cols] = torch.complex(*torch.randint(-3, 4, (2, n, cols), device='cuda', generator=g).float())
        return a, a[:, :cols].to(torch.complex128)

    dA, A = block(P, lda)
    dB, B = block(Q, ldb)
    ws = torch.empty(int(L.qdkp_block_gram_workspace_size(max(P, Q), max(P, Q))), dtype=torch.uint8, device='cuda')
    for d2, ld2, c2, B2 in ((dB, ldb, Q, B), (dA, lda, P, A)):      # A^H B, and A^H A
        assert -(-P // 12) * -(-c2 // 12) <= 16                      # else another kernel's
        out = np.empty((P, c2), dtype=np.complex128)
        _lib.check(L.qdkp_block_gram(dA.data_ptr(), lda, P, d2.data_ptr(), ld2, c2, n, _lib.C64,
                                     out.ctypes.data, ws.data_ptr(), ws.numel(), None), 'qdkp_block_gram')
        ref = (A.mH @ B2).cpu().numpy()
        assert np.array_equal(out, ref)


def test_workspace_of_a_wider_product_serves_narrower_ones():
    """qdkp_block_gram_workspace_size grows with either width: room for the widest product of a program is
    room for all of them."""
    from qd3dsolver_b200 import _lib
    size = _lib.lib().qdkp_block_gram_workspace_size
    w = np.array([[int(size(P, Q)) for Q in range(1, 73)] for P in range(1, 73)])
    assert (np.diff(w, axis=0) >= 0).all() and (np.diff(w, axis=1) >= 0).all()
