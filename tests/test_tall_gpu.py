"""The Gram and Ritz-update kernels where they can go wrong: rows that end inside a tile or a chunk, odd
widths and leading dimensions (copies of 8 bytes), a Hermitian product, panels of many warps, and
every accumulator count of the one-pass Ritz update."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('prec', ['c128', 'c64'])
@pytest.mark.parametrize('n, P, Q, lda, ldb', [
    (1, 1, 1, 1, 1), (7, 3, 2, 3, 2), (31, 12, 12, 12, 12), (33, 5, 24, 7, 24), (1023, 13, 1, 13, 3),
    (1024, 36, 24, 36, 24), (1025, 36, 36, 37, 36), (4099, 72, 72, 72, 72),
    (1030, 61, 51, 61, 51), (1031, 61, 51, 62, 51), (151_553, 12, 5, 12, 5)])
def test_gram_edges(n, P, Q, lda, ldb, prec):
    import torch
    from qd3dsolver_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(n + P)
    dt, code = (np.complex128, _lib.C128) if prec == 'c128' else (np.complex64, _lib.C64)

    def block(cols, ld):
        a = np.full((n, ld), np.nan, dt)
        a[:, :cols] = rng.standard_normal((n, cols)) + 1j * rng.standard_normal((n, cols))
        return torch.from_numpy(a).cuda(), a[:, :cols].astype(np.complex128)

    dA, A = block(P, lda)
    dB, B = block(Q, ldb)
    ws = torch.empty(int(L.qdkp_block_gram_workspace_size(max(P, Q), max(P, Q))),
                     dtype=torch.uint8, device='cuda')
    for d2, ld2, c2, B2 in ((dB, ldb, Q, B), (dA, lda, P, A)):      # A^H B, and A^H A
        if prec == 'c64' and -(-P // 12) * -(-c2 // 12) <= 16:
            continue        # a complex64 product that one CTA holds is another kernel's (split TF32)
        out = np.empty((P, c2), dtype=np.complex128)
        _lib.check(L.qdkp_block_gram(dA.data_ptr(), lda, P, d2.data_ptr(), ld2, c2, n, code,
                                     out.ctypes.data, ws.data_ptr(), ws.numel(), None),
                   'qdkp_block_gram')
        ref = A.conj().T @ B2
        # FP64 products of exact inputs: n + a few roundings of terms no larger than the scale, which
        # grow like sqrt(n); 1e-14 covers n = 2e5
        scale = (np.abs(A).T @ np.abs(B2)).max()
        assert np.abs(out - ref).max() / scale < 1e-14


# odd widths of complex64: its even ones run the paired H.X, which differs at the walls of the box
@pytest.mark.parametrize('phase, m', [('c128', m) for m in (1, 4, 5, 8, 12, 13, 16, 17, 20, 24)]
                         + [('c64', m) for m in (1, 5, 11, 13, 17, 23)])
def test_engine_iterates_follow_scipy(phase, m):
    import ctypes
    import scipy.sparse.linalg as spla
    import torch
    from qd3dsolver_b200 import _lib, kp_pryor as kpg, serving
    from qd3dsolver_b200.eigensolvers import start_block
    from oracle import kp_operator as ko
    keys = ('gamma1', 'gamma2', 'gamma3', 'P0', 'Ec', 'Ev', 'delta_so', 'b', 'd')
    strain = ('exx', 'eyy', 'ezz', 'exy', 'eyz', 'ezx')
    rng = np.random.default_rng(m)
    shape = (5, 7, 6)                       # 1680 rows: three parts of 512 and one of 144
    f = {k: rng.uniform(0.5, 3.0, shape) for k in keys}
    f.update({k: rng.uniform(-0.1, 0.1, shape) for k in strain})
    H = kpg.confined_hamiltonian(kpg.GridOperators(shape, 0.5), f, 8, strain={k: f[k] for k in strain})
    Ho = ko.confined_hamiltonian(shape, 0.5, f, 8, strain=True)
    its = 3
    r = serving.Request(H, k=m, extra=0, folded=False, tol=1e-12, maxiter=its, seed=m,
                        precision='mixed' if phase == 'c64' else 'c128', mixed_tol=1e-12)
    eng = serving.Engine(1)
    slot = eng.admit(r, phase=phase)
    eng.step(its + 2)
    lam = np.empty(m)
    V = torch.empty((H.shape[0], m), dtype=torch.complex128, device='cuda')
    res = np.empty(m)
    info = _lib.LobpcgInfo()
    _lib.check(_lib.lib().qdkp_engine_retire(eng._h, slot, lam.ctypes.data, V.data_ptr(),
                                             res.ctypes.data, ctypes.byref(info), eng.stream), 'retire')
    eng.close()
    with warnings.catch_warnings():
        warnings.simplefilter('ignore')
        mu, _ = spla.lobpcg(Ho, start_block(H.shape[0], m, m, True), largest=False, tol=1e-12,
                            maxiter=its)
    # rounding of the blocks against |H|, grown by the Cholesky orthonormalisations of R and P
    # (condition numbers of some 10 an iteration over three iterations): 1e3 of the unit
    eps = np.finfo(np.float64 if phase == 'c128' else np.float32).eps
    bound = 1e3 * eps * spla.norm(Ho, 1)
    assert np.abs(np.sort(lam) - np.sort(mu)).max() < bound
    # the returned block carries those values: V^H H V = diag(lambda)
    Vh = V.cpu().numpy()
    assert np.abs(Vh.conj().T @ (Ho @ Vh) - np.diag(lam)).max() < bound
    H.close()


@pytest.mark.parametrize('kind', ['random', 'pairs', 'diagonal', 'identity', 'zero'])
@pytest.mark.parametrize('n', [1, 2, 3, 5, 8, 13, 16, 23, 24])
def test_eigh_all_pairs_of_a_block(n, kind):
    """All pairs of a matrix of a block's width: the widths the multisection route takes, with spectra
    that split the tridiagonal (diagonal, identity, zero) and exactly degenerate pairs."""
    import torch
    from qd3dsolver_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(n)
    Q, _ = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    lam = {'random': rng.uniform(-1, 1, n), 'pairs': np.repeat(np.arange(n // 2 + 1) + 0.5, 2)[:n],
           'diagonal': rng.uniform(-1, 1, n), 'identity': np.ones(n), 'zero': np.zeros(n)}[kind]
    A = np.diag(lam).astype(np.complex128) if kind in ('diagonal', 'identity', 'zero') else (Q * lam) @ Q.conj().T
    A = np.ascontiguousarray((A + A.conj().T) / 2)
    ws = torch.empty(int(L.qdkp_block_eigh_workspace_size(n)), dtype=torch.uint8, device='cuda')
    w, V = np.zeros(n), np.zeros((n, n), dtype=np.complex128)
    _lib.check(L.qdkp_block_eigh(A.ctypes.data, None, n, n, w.ctypes.data, V.ctypes.data, ws.data_ptr(),
                                 ws.numel(), None), 'qdkp_block_eigh')
    # a backward-stable eigensolve: a modest multiple of n rounding units of the norm
    tol = 50 * n * np.finfo(float).eps * max(1.0, np.abs(lam).max())
    assert np.all(np.diff(w) >= 0)
    assert np.abs(w - np.sort(lam)).max() <= tol
    assert np.abs(A @ V - V * w).max() <= tol
    assert np.abs(V.conj().T @ V - np.eye(n)).max() <= tol


@pytest.mark.parametrize('m, a, b', [(2, 0, 1), (6, 1, 3), (12, 0, 11), (13, 11, 12), (24, 7, 16)])
def test_repeated_columns_are_refused(m, a, b):
    """A start block with a repeated column: the pivot is rounding noise of either sign."""
    import torch
    from qd3dsolver_b200 import _lib, kp_pryor as kpg, serving
    from qd3dsolver_b200.eigensolvers import lobpcg_device, start_block
    keys = ('gamma1', 'gamma2', 'gamma3', 'P0', 'Ec', 'Ev', 'delta_so', 'b', 'd')
    shape = (5, 7, 6)
    H = kpg.confined_hamiltonian(kpg.GridOperators(shape, 0.5), {k: np.ones(shape) for k in keys}, 8)
    for seed in range(4):
        X0 = start_block(H.shape[0], m, seed, True)
        X0[:, b] = X0[:, a]
        with pytest.raises(_lib.QdkpError, match='Linearly dependent initial approximations'):
            lobpcg_device(H, X0, folded=False, sigma=0.0, tol=1e-9, maxiter=2)
        eng = serving.Engine(1)
        r = serving.Request(H, k=m, extra=0, folded=False, maxiter=2)
        with pytest.raises(_lib.QdkpError, match='Linearly dependent initial approximations'):
            eng.admit(r, X0=torch.from_numpy(X0).cuda())
        eng.close()
    H.close()
