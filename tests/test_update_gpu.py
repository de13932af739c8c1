"""Block updates Y = A C where the rows or the columns end inside what a warp or a CTA takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one tile, either span (64 and 128 rows) and the grid's 592 CTAs of each, a row short or long
@pytest.mark.parametrize('n', [1, 9, 63, 64, 65, 127, 129, 592 * 64 - 1, 592 * 64 + 1, 592 * 128 + 1])
@pytest.mark.parametrize('prec, P, q', [('c128', 36, 12), ('c128', 39, 13), ('c128', 23, 24), ('c128', 72, 24),
                                        ('c64', 21, 7), ('c64', 51, 17), ('c64', 72, 24)])
def test_updates_at_the_edges_of_their_spans(n, prec, P, q):
    import torch
    from qd3dsolver_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(n + P)
    dt, code, tol = (torch.complex128, _lib.C128, 1e-14) if prec == 'c128' else (torch.complex64, _lib.C64, 1e-6)
    lda, ldy = P + 2, q + 1
    A = torch.full((n, lda), float('nan'), dtype=dt, device='cuda')
    a = torch.randn((n, P), dtype=dt, device='cuda', generator=torch.Generator('cuda').manual_seed(n))
    A[:, :P] = a
    C = rng.standard_normal((P, q)) + 1j * rng.standard_normal((P, q))
    Cd = torch.from_numpy(C).cuda()
    Y = torch.full((n, ldy), 7.0, dtype=dt, device='cuda')
    ws = torch.empty(int(L.qdkp_block_update_workspace_size(P, q)), dtype=torch.uint8, device='cuda')
    _lib.check(L.qdkp_block_update(A.data_ptr(), lda, P, C.ctypes.data, q, n, Y.data_ptr(), ldy, code,
                                   ws.data_ptr(), ws.numel(), None), 'qdkp_block_update')
    ref = a.to(torch.complex128) @ Cd
    # P products, and in complex64 their factors in 22 bits, against the sum of their moduli
    scale = float((a.to(torch.complex128).abs() @ Cd.abs()).max())
    assert float((Y[:, :q] - ref).abs().max()) < tol * scale
    assert bool((Y[:, q:] == 7.0).all())
