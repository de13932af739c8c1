"""A raised fault flag (a kernel's bounded wait gave up) reaches the caller of every entry point that waits for
such kernels, and is gone once cleared. The flag is raised on the host; no GPU fault is involved."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ('gamma1', 'gamma2', 'gamma3', 'P0', 'Ec', 'Ev', 'delta_so', 'b', 'd')


def test_raised_flag_reaches_every_caller():
    import torch
    from qd3dsolver_b200 import _lib, eigensolvers as eg, kp_pryor as kpg, serving
    L = _lib.lib()
    rng = np.random.default_rng(0)
    shape = (5, 7, 6)
    H = kpg.confined_hamiltonian(kpg.GridOperators(shape, 0.5),
                                 {k: rng.uniform(0.5, 3.0, shape) for k in KEYS}, 8)
    n, m = H.shape[0], 4
    X = torch.randn((n, m), dtype=torch.complex128, device='cuda', generator=torch.Generator('cuda').manual_seed(0))
    X0 = eg.start_block(n, m, 0, True)
    out = np.empty((m, m), dtype=np.complex128)
    C = np.eye(m, dtype=np.complex128)
    Y = torch.empty_like(X)
    ws = torch.empty(max(int(L.qdkp_block_gram_workspace_size(m, m)), int(L.qdkp_block_update_workspace_size(m, m))),
                     dtype=torch.uint8, device='cuda')

    def gram():
        _lib.check(L.qdkp_block_gram(X.data_ptr(), m, m, X.data_ptr(), m, m, n, _lib.C128, out.ctypes.data,
                                     ws.data_ptr(), ws.numel(), None), 'qdkp_block_gram')

    def update():
        _lib.check(L.qdkp_block_update(X.data_ptr(), m, m, C.ctypes.data, m, n, Y.data_ptr(), m, _lib.C128,
                                       ws.data_ptr(), ws.numel(), None), 'qdkp_block_update')

    def noalloc():
        _lib.check(L.qdkp_apply_folded_noalloc(H.handle, X.data_ptr(), m, Y.data_ptr(), m, m, 0.5, _lib.C128,
                                               torch.cuda.current_stream().cuda_stream), 'noalloc')

    eng = serving.Engine(2)
    request = lambda: serving.Request(H, k=m, extra=0, folded=False, tol=1e-9, maxiter=5)
    resident = eng.admit(request())
    eng.step(2)
    calls = dict(
        apply=lambda: H.apply(X), host=lambda: H.apply_host(X0), noalloc=noalloc, gram=gram, update=update,
        solve=lambda: eg.lobpcg_device(H, X0, folded=False, sigma=0.0, tol=1e-9, maxiter=2),
        residuals=lambda: eg.residual_norms(H, np.zeros(m), X0),
        admit=lambda: eng.admit(request()), step=lambda: eng.step(1), poll=eng.poll)

    def flag(clear):
        f = ctypes.c_int(-1)
        assert L.qdkp_device_fault(torch.cuda.current_device(), clear, ctypes.byref(f)) == 0
        return f.value

    assert flag(0) == 0
    assert L.qdkp_device_fault_inject(torch.cuda.current_device()) == 0
    try:
        for name, call in calls.items():
            with pytest.raises(_lib.QdkpError, match='gave up waiting'):
                call()
                pytest.fail(f'{name} did not report the flag')
        with pytest.raises(_lib.QdkpError, match='gave up waiting'):
            eng.retire(resident)
        assert flag(0) == 1
    finally:
        assert flag(1) == 1
    assert flag(0) == 0
    for name, call in calls.items():
        call()
    assert np.allclose(out, (X.mH @ X).cpu().numpy(), rtol=0, atol=1e-10)
    eng.close()
    H.close()
