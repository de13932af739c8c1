"""H.X tile shapes where they can go wrong, against the oracle CSR: grids that end inside a tile, on
its edge or one site past it, one or two planes along x, column counts below, at and past a
tile's columns, odd leading dimensions, and the band slices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ('gamma1', 'gamma2', 'gamma3', 'P0', 'Ec', 'Ev', 'delta_so', 'b', 'd')
STRAIN = ('exx', 'eyy', 'ezz', 'exy', 'eyz', 'ezx')


def _fields(shape, rng):
    f = {k: rng.uniform(0.5, 3.0, shape) for k in KEYS}
    f.update({k: rng.uniform(-0.1, 0.1, shape) for k in STRAIN})
    return f


@pytest.mark.parametrize('bands', [8, 6, 4])
@pytest.mark.parametrize('shape', [(1, 10, 10), (2, 6, 10), (5, 11, 14), (9, 16, 24), (3, 17, 25),
                                   (20, 9, 9), (4, 1, 3)])
def test_tiles_at_their_edges(shape, bands):
    import torch
    from qd3dsolver_b200 import _lib, kp_pryor as kpg
    from oracle import kp_operator as ko
    rng = np.random.default_rng(sum(shape) + bands)
    f = _fields(shape, rng)
    hole = bands != 8
    H = kpg.confined_hamiltonian(kpg.GridOperators(shape, 0.5), f, bands, hole_convention=hole,
                                 strain={k: f[k] for k in STRAIN})
    Ho = ko.confined_hamiltonian(shape, 0.5, f, bands, hole_convention=hole, strain=True)
    n = H.shape[0]
    X = rng.standard_normal((n, 17)) + 1j * rng.standard_normal((n, 17))
    ref = Ho @ X
    scale = np.abs(ref).max()
    for dt, code, tol, tiles in ((torch.complex128, _lib.C128, 1e-13, 4),
                                 (torch.complex64, _lib.C64, 2e-6, _lib.TILE_COUNT)):
        Xd = torch.from_numpy(X).cuda().to(dt)
        for tile in list(range(tiles)) + [_lib.TILE_DIRECT, _lib.TILE_AUTO]:
            H.set_tile(tile, code)
            for m, ld in ((1, 1), (2, 2), (3, 4), (4, 4), (5, 5), (8, 8), (12, 13), (17, 18)):
                big = torch.full((n, ld), float('nan'), dtype=dt, device='cuda')
                big[:, :m] = Xd[:, :m]
                out = torch.full((n, ld), 7.0, dtype=dt, device='cuda')
                H.apply(big[:, :m], out=out[:, :m])
                err = np.abs(out[:, :m].cpu().numpy() - ref[:, :m]).max() / scale
                assert err < tol, (tile, m, ld, err)
                assert bool((out[:, m:] == 7.0).all()), (tile, m, ld)
    H.close()


@pytest.mark.parametrize('bands', [8, 6, 4])
@pytest.mark.parametrize('shape', [(1, 10, 10), (5, 11, 14), (9, 16, 24), (4, 1, 3)])
def test_folded_passes_its_block_uncoupled(shape, bands):
    """(H - sigma)^2 X through every kernel that its two applies can take, against the oracle CSR."""
    import torch
    from qd3dsolver_b200 import _lib, kp_pryor as kpg
    from oracle import kp_operator as ko
    rng = np.random.default_rng(sum(shape) + bands)
    f = _fields(shape, rng)
    hole = bands != 8
    H = kpg.confined_hamiltonian(kpg.GridOperators(shape, 0.5), f, bands, hole_convention=hole,
                                 strain={k: f[k] for k in STRAIN})
    Ho = ko.confined_hamiltonian(shape, 0.5, f, bands, hole_convention=hole, strain=True)
    n = H.shape[0]
    X = rng.standard_normal((n, 13)) + 1j * rng.standard_normal((n, 13))
    sigma = 0.7
    T = Ho @ X - sigma * X
    ref = Ho @ T - sigma * T
    scale = np.abs(ref).max()
    # two applies, each with the rounding of one (the tolerances above)
    for dt, code, tol, tiles in ((torch.complex128, _lib.C128, 2e-13, 4),
                                 (torch.complex64, _lib.C64, 4e-6, 6)):
        Xd = torch.from_numpy(X).cuda().to(dt)
        for tile in list(range(tiles)) + [_lib.TILE_DIRECT, _lib.TILE_AUTO]:
            H.set_tile(tile, code)
            for m in (1, 3, 4, 8, 13):
                out = H.apply(Xd[:, :m].contiguous(), sigma=sigma, mode=_lib.APPLY_FOLDED)
                err = np.abs(out.cpu().numpy() - ref[:, :m]).max() / scale
                assert err < tol, (tile, m, err)
    H.close()
