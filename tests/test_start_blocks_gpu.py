"""Which start blocks a solve takes: a repeated column is refused, one that differs by more than the rounding of
the Gram matrix is a column of its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m, a, b', [(2, 0, 1), (6, 1, 3), (12, 0, 11)])
def test_nearly_repeated_columns(m, a, b):
    """Seeded blocks with a column 3e-8 off another (relative): their pivots, 9e-16 of the diagonal give or take
    the sums' rounding, are positive, which was all that was asked of them before repeated columns were refused
    whichever way their pivot rounds."""
    from qd3dsolver_b200 import _lib, kp_pryor as kpg
    from qd3dsolver_b200.eigensolvers import lobpcg_device, start_block
    keys = ('gamma1', 'gamma2', 'gamma3', 'P0', 'Ec', 'Ev', 'delta_so', 'b', 'd')
    shape = (9, 8, 7)
    H = kpg.confined_hamiltonian(kpg.GridOperators(shape, 0.5), {k: np.ones(shape) for k in keys}, 8)
    n = H.shape[0]
    solve = lambda X: lobpcg_device(H, X, folded=False, sigma=0.0, tol=1e-9, maxiter=1)
    for seed in range(12):
        rng = np.random.default_rng(seed)
        X0 = start_block(n, m, seed, True)
        x = X0[:, a].copy()
        z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        X0[:, b] = x + 3e-8 * z * np.linalg.norm(x) / np.linalg.norm(z)
        solve(X0)
        for factor in (1.0, 2.0, 0.5):
            X0[:, b] = factor * x
            with pytest.raises(_lib.QdkpError, match='Linearly dependent initial approximations'):
                solve(X0)
    H.close()
