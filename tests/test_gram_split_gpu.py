"""How the rows of a Gram product are split: edges of the parts, and short blocks that have to fill the GPU."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gram(L, _lib, dA, P, dB, Q, code, ws):
    out = np.empty((P, Q), dtype=np.complex128)
    _lib.check(L.qdkp_block_gram(dA.data_ptr(), P, P, dB.data_ptr(), Q, Q, dA.shape[0], code,
                                 out.ctypes.data, ws.data_ptr(), ws.numel(), None), 'qdkp_block_gram')
    return out


# one part, two, the most short ones with a full, a short or an empty last one, and where longer parts begin
@pytest.mark.parametrize('n', [127, 128, 255, 256, 257, 5000, 9471, 9472, 9473, 18945, 75775, 75777])
@pytest.mark.parametrize('prec, P, Q', [('c128', 12, 5), ('c128', 39, 26), ('c64', 61, 51)])
def test_parts_at_their_edges(n, prec, P, Q):
    import torch
    from qd3dsolver_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(n + P)
    dt, code = (np.complex128, _lib.C128) if prec == 'c128' else (np.complex64, _lib.C64)
    A = (rng.standard_normal((n, P)) + 1j * rng.standard_normal((n, P))).astype(dt)
    B = (rng.standard_normal((n, Q)) + 1j * rng.standard_normal((n, Q))).astype(dt)
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    ws = torch.empty(int(L.qdkp_block_gram_workspace_size(P, P)), dtype=torch.uint8, device='cuda')
    A, B = A.astype(np.complex128), B.astype(np.complex128)
    for d2, B2, c2 in ((dB, B, Q), (dA, A, P)):
        out = _gram(L, _lib, dA, P, d2, c2, code, ws)
        # FP64 sums of exact inputs: roundings grow like sqrt(n); 1e-14 covers n = 2e4
        assert np.abs(out - A.conj().T @ B2).max() < 1e-14 * (np.abs(A).T @ np.abs(B2)).max()


def test_a_short_block_takes_a_share_of_a_long_ones_time():
    """20,000 rows of 39 x 26 columns against 150,000: with a thousand rows a part a product of any length up
    to 151,552 rows took the same 100 - 110 us; spread over all SMs the short one takes 50."""
    import torch
    from qd3dsolver_b200 import _lib
    L = _lib.lib()
    P, Q = 39, 26
    ws = torch.empty(int(L.qdkp_block_gram_workspace_size(P, Q)), dtype=torch.uint8, device='cuda')

    def best(n):
        dA = torch.ones((n, P), dtype=torch.complex128, device='cuda')
        dB = torch.ones((n, Q), dtype=torch.complex128, device='cuda')
        times = []
        for _ in range(40):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            _gram(L, _lib, dA, P, dB, Q, _lib.C128, ws)
            times.append(time.perf_counter() - t0)
        return min(times)
    assert best(20_000) < 0.65 * best(150_000)


def test_leading_dimension_beyond_32_bits():
    """Two rows that lie 2^31 + 8 elements apart (17 GB)."""
    import torch
    from qd3dsolver_b200 import _lib
    L = _lib.lib()
    P, Q, ld = 61, 51, 2 ** 31 + 8
    a = torch.empty(ld + P, dtype=torch.complex64, device='cuda')
    A = torch.randn((2, P), dtype=torch.complex64, device='cuda', generator=torch.Generator('cuda').manual_seed(1))
    a[:P], a[ld:] = A[0], A[1]
    B = A[:, :Q].contiguous()
    ws = torch.empty(int(L.qdkp_block_gram_workspace_size(P, Q)), dtype=torch.uint8, device='cuda')
    out = np.empty((P, Q), dtype=np.complex128)
    _lib.check(L.qdkp_block_gram(a.data_ptr(), ld, P, B.data_ptr(), Q, Q, 2, _lib.C64, out.ctypes.data,
                                 ws.data_ptr(), ws.numel(), None), 'qdkp_block_gram')
    A = A.to(torch.complex128).cpu().numpy()
    # two products an entry, in FP64
    assert np.abs(out - A.conj().T @ A[:, :Q]).max() < 1e-14 * (np.abs(A).T @ np.abs(A)).max()
