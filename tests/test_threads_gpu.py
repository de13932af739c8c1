"""Calls of different sizes from several threads, each on a stream of its own."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_eigensolves_of_different_widths_at_once():
    """A kernel's shared-memory limit belongs to the process: a narrow matrix on one thread must not lower it
    under a wide one's launch on another (of one size class: 41 to 64 rows)."""
    import torch
    from qd3dsolver_b200 import _lib
    L = _lib.lib()
    errors = []

    def work(n, calls):
        torch.cuda.set_device(0)
        st = torch.cuda.Stream()
        rng = np.random.default_rng(n)
        a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        A = np.ascontiguousarray((a + a.conj().T) / 2)
        ref = np.linalg.eigvalsh(A)
        ws = torch.empty(int(L.qdkp_block_eigh_workspace_size(n)), dtype=torch.uint8, device='cuda')
        w, V = np.zeros(n), np.zeros((n, n), dtype=np.complex128)
        try:
            for _ in range(calls):
                _lib.check(L.qdkp_block_eigh(A.ctypes.data, None, n, n // 3, w.ctypes.data, V.ctypes.data, ws.data_ptr(),
                                             ws.numel(), st.cuda_stream), f'n = {n}')
                assert np.abs(w[:n // 3] - ref[:n // 3]).max() < 1e-12 * np.abs(ref).max()
        except Exception as e:                              # noqa: BLE001 -- reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(n, 400)) for n in (64, 41, 64, 42)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
