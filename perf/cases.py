"""The work this library is used for, as timed cases.

Each case is one call, or one short run of calls, that a program makes through the package's
entry points, on operators of square-based InAs pyramids in GaAs:

  apply     H X, (H - sigma) X or (H - sigma)^2 X on a device block (`KPOperator.apply`), in
            complex128 and complex64, eight- and six-band
  solve     a budget of iterations of the single-solve drop-in (`eigensolvers.lobpcg_device`)
  serve     the batched engine (`serving.Engine`): admit every solve of a dot-size sweep, run a
            budget of ticks, retire them, in the complex128 form or the complex64 search
  ritz      the block products of one Rayleigh-Ritz step through the C ABI: the Gram matrix
            [X R P]^H [AR AP] and the update [X R P] C
  strain    inhomogeneous elasticity of a dot (`fields.solve_strain_fd`)

`listed()` are the cases to time, `draw(rng)` gives more of the same ranges, `prepare` makes what
a program has in hand before the call, `run` is one pass, `work` what a pass cannot do without
and `exact` its result in 64 bits, in plain torch.
"""
import math

import numpy as np
import torch

from qd3dsolver_b200 import _lib, eigensolvers, fields, kp_pryor, serving

G = 0.0380998                     # hbar^2 / 2 m0 in eV nm^2
STRAIN = ('exx', 'eyy', 'ezz', 'exy', 'eyz', 'ezx')
#: Pryor's Table I for InAs (inside the dot) and GaAs (outside).
INAS = dict(gamma1L=19.67, gamma2L=8.37, gamma3L=9.29, Eg=0.418, delta_so=0.38, Ep=22.2,
            a_c=-6.66, a_v=0.66, b=-1.8, d=-3.6, C=(83.29, 45.26, 39.59), a0=6.0583, vbo=0.085)
GAAS = dict(gamma1L=6.85, gamma2L=2.1, gamma3L=2.9, Eg=1.519, delta_so=0.33, Ep=25.7,
            a_c=-9.3, a_v=0.7, b=-2.0, d=-5.4, C=(121.1, 54.8, 60.4), a0=5.6532, vbo=0.0)
#: Grids of the dot-size sweep: bases 6 ... 18 nm at 1 nm spacing with 8 nm of matrix around.
SWEEP = ((23, 20), (25, 21), (27, 22), (29, 23), (31, 24), (33, 25), (35, 26))


def listed():
    return [
        # one vector on a small dot: what a norm estimate, a Hermiticity probe or a caller's own
        # Lanczos does many times, bound by the launch
        dict(name='matvec_c128', kind='apply', nxy=23, nz=20, h=1.0, bands=8, m=1,
             dtype='c128', mode='plain'),
        # the operator of the folded solves of a 10 nm dot, the block an 8-state solve uses
        dict(name='folded_c128_27', kind='apply', nxy=27, nz=22, h=1.0, bands=8, m=12,
             dtype='c128', mode='folded'),
        # the same in the search precision on the 24 x 24 x 18 nm box at 0.5 nm
        dict(name='folded_c64_48', kind='apply', nxy=48, nz=36, h=0.5, bands=8, m=12,
             dtype='c64', mode='folded'),
        # the full-size dot (48 x 48 x 36 nm at 0.375 nm), eight Kramers pairs and guard vectors
        dict(name='apply_c128_128', kind='apply', nxy=128, nz=96, h=0.375, bands=8, m=24,
             dtype='c128', mode='plain'),
        dict(name='apply_c64_128', kind='apply', nxy=128, nz=96, h=0.375, bands=8, m=24,
             dtype='c64', mode='plain'),
        # the six-band hole route of a thick matrix box
        dict(name='apply_six_band', kind='apply', nxy=47, nz=41, h=0.5, bands=6, m=12,
             dtype='c128', mode='plain'),
        # the single-solve drop-in on a 10 nm dot, and on the 0.5 nm grid
        dict(name='solve_27', kind='solve', nxy=27, nz=22, h=1.0, m=12, iters=10),
        dict(name='solve_48', kind='solve', nxy=48, nz=36, h=0.5, m=12, iters=8),
        # both bands of all seven dots of the sweep resident at once, finish and search precision
        dict(name='sweep_c128', kind='serve', dots=7, k=8, ticks=8, phase='c128'),
        dict(name='sweep_c64', kind='serve', dots=7, k=8, ticks=4, phase='c64'),
        # the block products of one iteration on the 0.5 nm grid
        dict(name='ritz_c128', kind='ritz', n=663552, m=12, dtype='c128'),
        # elasticity of a buried dot, as every environment is built
        dict(name='strain_96', kind='strain', nxy=96, nz=72, h=0.5),
    ]


def _spread(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(('apply', 'apply', 'solve', 'serve', 'ritz', 'strain'))
    if kind == 'apply':
        bands = rng.choice((8, 8, 8, 6, 4))
        nxy = _spread(rng, 14, 112)
        return dict(kind='apply', nxy=nxy, nz=max(12, int(nxy * rng.uniform(0.6, 1.0))),
                    h=rng.choice((0.375, 0.5, 1.0)), bands=bands, m=_spread(rng, 1, 24),
                    dtype=rng.choice(('c128', 'c64')),
                    mode=rng.choice(('plain', 'shifted', 'folded')))
    if kind == 'solve':
        nxy = _spread(rng, 14, 48)
        return dict(kind='solve', nxy=nxy, nz=max(12, int(nxy * rng.uniform(0.6, 0.9))),
                    h=rng.choice((0.5, 1.0)), m=rng.randint(6, 24), iters=rng.randint(4, 8))
    if kind == 'serve':
        # few ticks in complex64: Ritz vectors of close values mix by rounding as they go on
        phase = rng.choice(('c128', 'c64'))
        return dict(kind='serve', dots=rng.randint(1, 7), k=2 * rng.randint(2, 4),
                    ticks=rng.randint(4, 8) if phase == 'c128' else rng.randint(2, 4), phase=phase)
    if kind == 'ritz':
        return dict(kind='ritz', n=_spread(rng, 20000, 650000), m=rng.randint(6, 24),
                    dtype=rng.choice(('c128', 'c64')))
    nxy = _spread(rng, 20, 96)
    return dict(kind='strain', nxy=nxy, nz=max(16, int(nxy * rng.uniform(0.6, 0.75))),
                h=rng.choice((0.375, 0.5, 1.0)))


# --------------------------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------------------------

def _mask(nxy, nz, h, rng):
    """Square {101} pyramid of a seeded size standing in the lower half of the box."""
    base = nxy * h * rng.uniform(0.33, 0.42)
    c = (np.arange(nxy) - (nxy - 1) / 2.0) * h
    z = (np.arange(nz) - int(0.3 * nz) + 0.5) * h
    half = base / 2.0 - z
    return ((z >= 0.0) & (half > 0.0))[None, None, :] & \
        (np.abs(c)[:, None, None] < half) & (np.abs(c)[None, :, None] < half)


def _fourier_strain(mask, h):
    """Elastic strain of the dot in a homogeneous GaAs matrix (one FFT, Christoffel inverse)."""
    C11, C12, C44 = GAAS['C']
    eT = -(GAAS['a0'] - INAS['a0']) / INAS['a0']
    chi = torch.from_numpy(mask).cuda().double()
    ck = torch.fft.fftn(chi)
    k = torch.meshgrid(*[2 * math.pi * torch.fft.fftfreq(n, d=h, dtype=torch.float64,
                                                         device='cuda') for n in mask.shape],
                       indexing='ij')
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    M = [[(C12 + C44) * k[i] * k[j] + ((C11 - C12 - 2 * C44) * k[i] ** 2 + C44 * k2
                                       if i == j else 0.0) for j in range(3)] for i in range(3)]
    cof = [[M[(i + 1) % 3][(j + 1) % 3] * M[(i + 2) % 3][(j + 2) % 3]
            - M[(i + 1) % 3][(j + 2) % 3] * M[(i + 2) % 3][(j + 1) % 3] for j in range(3)]
           for i in range(3)]
    det = sum(M[0][j] * cof[0][j] for j in range(3))
    inv = torch.where(det != 0.0, 1.0 / torch.where(det != 0.0, det, 1.0), 0.0)
    u = [-1j * eT * (C11 + 2 * C12) * ck * inv * sum(cof[i][j] * k[j] for j in range(3))
         for i in range(3)]

    def back(i, j):
        e = torch.fft.ifftn(0.5j * (k[i] * u[j] + k[j] * u[i])).real
        return (e - eT * chi if i == j else e).cpu().numpy()
    return dict(exx=back(0, 0), eyy=back(1, 1), ezz=back(2, 2), exy=back(0, 1), eyz=back(1, 2),
                ezx=back(2, 0))


def _environment(nxy, nz, h, bands, seed):
    """(coefficient fields with strain, conduction sigma, valence sigma) of one seeded dot."""
    rng = np.random.default_rng(seed)
    mask = _mask(nxy, nz, h, rng)
    st = _fourier_strain(mask, h)

    def pick(key):
        return np.where(mask, INAS[key], GAAS[key])
    tr = st['exx'] + st['eyy'] + st['ezz']
    Ev0 = pick('vbo')
    f = dict(st, Ec=Ev0 + pick('Eg') + pick('a_c') * tr, Ev=Ev0 - pick('a_v') * tr,
             delta_so=pick('delta_so'), b=pick('b'), d=pick('d'))
    shift = [m['Ep'] / (3 * m['Eg'] + m['delta_so']) if bands == 8 else 0.0 for m in (INAS, GAAS)]
    for key, part in (('gamma1', 1.0), ('gamma2', 0.5), ('gamma3', 0.5)):
        f[key] = np.where(mask, INAS[key + 'L'] - part * shift[0], GAAS[key + 'L'] - part * shift[1])
    f['P0'] = np.sqrt(pick('Ep') * G)
    return f, float(f['Ec'][mask].min()), float(f['Ev'][mask].max()) + 0.1


def _operator(nxy, nz, h, bands, seed):
    f, se, sv = _environment(nxy, nz, h, bands, seed)
    ops = kp_pryor.GridOperators((nxy, nxy, nz), h)
    H = kp_pryor.confined_hamiltonian(ops, f, bands, hole_convention=bands != 8,
                                      strain={k: f[k] for k in STRAIN})
    return H, se, sv


def _block(n, m, seed, dtype=torch.complex128):
    g = torch.Generator(device='cuda').manual_seed(seed)
    return torch.randn((n, m), dtype=dtype, device='cuda', generator=g)


def _ritz_inputs(case, seed):
    n, m = case['n'], case['m']
    dt = torch.complex128 if case['dtype'] == 'c128' else torch.complex64
    W = _block(n, 3 * m, seed, dt)
    A = _block(n, 2 * m, seed + 1, dt)
    rng = np.random.default_rng(seed)
    C = rng.standard_normal((3 * m, m)) + 1j * rng.standard_normal((3 * m, m))
    return W, A, C


_MODES = dict(plain=_lib.APPLY_PLAIN, shifted=_lib.APPLY_SHIFTED, folded=_lib.APPLY_FOLDED)


def prepare(case, seed):
    kind = case['kind']
    if kind == 'apply':
        H, se, _ = _operator(case['nxy'], case['nz'], case['h'], case['bands'], seed)
        dt = torch.complex128 if case['dtype'] == 'c128' else torch.complex64
        X = _block(H.shape[0], case['m'], seed, dt)
        ws = torch.empty_like(X) if case['mode'] == 'folded' else None
        return dict(kind=kind, H=H, X=X, out=torch.empty_like(X), ws=ws, sigma=se,
                    mode=_MODES[case['mode']])
    if kind == 'solve':
        H, se, _ = _operator(case['nxy'], case['nz'], case['h'], 8, seed)
        return dict(kind=kind, H=H, X0=_block(H.shape[0], case['m'], seed), sigma=se,
                    iters=case['iters'])
    if kind == 'serve':
        solves = []
        for i, (nxy, nz) in enumerate(SWEEP[:case['dots']]):
            H, se, sv = _operator(nxy, nz, 1.0, 8, seed + i)
            block = case['k'] + max(2, case['k'] // 2)
            for j, s in enumerate((se, sv)):
                solves.append((H, s, _block(H.shape[0], block, seed + 100 + 2 * i + j)))
        return dict(kind=kind, solves=solves, engine=serving.Engine(max_slots=len(solves)),
                    k=case['k'], ticks=case['ticks'], phase=case['phase'])
    if kind == 'ritz':
        W, A, C = _ritz_inputs(case, seed)
        P, Q, q = W.shape[1], A.shape[1], C.shape[1]
        need = max(int(_lib.lib().qdkp_block_gram_workspace_size(P, Q)),
                   int(_lib.lib().qdkp_block_update_workspace_size(P, q)))
        return dict(kind=kind, W=W, A=A, C=C, gram=np.empty((P, Q), dtype=np.complex128),
                    Y=torch.empty((W.shape[0], q), dtype=W.dtype, device='cuda'),
                    ws=torch.empty(need, dtype=torch.uint8, device='cuda'))
    # an InAs-rich dot: the misfit goes with its composition
    rng = np.random.default_rng(seed)
    return dict(kind=kind, mask=_mask(case['nxy'], case['nz'], case['h'], rng), h=case['h'],
                misfit=(GAAS['a0'] - INAS['a0']) / INAS['a0'] * rng.uniform(0.6, 1.0))


# --------------------------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------------------------

def _density(V):
    """|psi|^2 per row and state: what is plotted and fed to a potential; a state's phase is
    arbitrary, its density is not."""
    return torch.view_as_real(V).square().sum(-1)


def run(s):
    kind = s['kind']
    if kind == 'apply':
        return s['H'].apply(s['X'], sigma=s['sigma'], mode=s['mode'], out=s['out'],
                            workspace=s['ws'])
    if kind == 'solve':
        lam, V, hist, _ = eigensolvers.lobpcg_device(s['H'], s['X0'], folded=True,
                                                     sigma=s['sigma'], tol=1e-9,
                                                     maxiter=s['iters'])
        return dict(ritz=lam, residuals=hist, density=_density(V))
    if kind == 'serve':
        eng, phase = s['engine'], s['phase']
        slots = []
        for H, sigma, X0 in s['solves']:
            r = serving.Request(H, k=s['k'], sigma=sigma, tol=1e-9, maxiter=s['ticks'] + 10,
                                precision='c128' if phase == 'c128' else 'mixed')
            slots.append(eng.admit(r, X0=X0, phase=phase))
        eng.step(s['ticks'])
        eng.poll()
        done = [eng.retire(slot).result for slot in slots]
        # the search phase's results carry its precision
        ft = np.float64 if phase == 'c128' else np.float32
        dt = torch.float64 if phase == 'c128' else torch.float32
        return dict(energies=np.concatenate([d['E'] for d in done]).astype(ft),
                    density=[_density(d['V']).to(dt) for d in done])
    if kind == 'ritz':
        W, A, C, Y, L = s['W'], s['A'], s['C'], s['Y'], _lib.lib()
        n, P, Q, q = W.shape[0], W.shape[1], A.shape[1], C.shape[1]
        prec = _lib.C128 if W.dtype == torch.complex128 else _lib.C64
        st = torch.cuda.current_stream().cuda_stream
        _lib.check(L.qdkp_block_gram(W.data_ptr(), P, P, A.data_ptr(), Q, Q, n, prec,
                                     s['gram'].ctypes.data, s['ws'].data_ptr(), s['ws'].numel(),
                                     st), 'qdkp_block_gram')
        _lib.check(L.qdkp_block_update(W.data_ptr(), P, P, C.ctypes.data, q, n, Y.data_ptr(), q,
                                       prec, s['ws'].data_ptr(), s['ws'].numel(), st),
                   'qdkp_block_update')
        return dict(gram=s['gram'].copy(), update=Y)
    e = fields.solve_strain_fd(s['mask'], s['misfit'], INAS['C'], GAAS['C'], s['h'], device=True)
    return [getattr(e, k) for k in STRAIN]


# --------------------------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------------------------

# real multiply-adds of one site and column: a Hermitian 8 x 8 (6 x 6, 4 x 4) block at the site
# and at its faces, the six valence bands at its edges, as real weights on complex values
_FMA = {8: 400, 6: 230, 4: 180}


def work(case):
    kind = case['kind']
    if kind == 'apply':
        N, m, nb = case['nxy'] ** 2 * case['nz'], case['m'], case['bands']
        s = 16 if case['dtype'] == 'c128' else 8
        times = 2 if case['mode'] == 'folded' else 1
        return dict(bytes=times * N * (15 * s / 2 + 2 * nb * m * s),
                    flops=times * 2.0 * _FMA[nb] * N * m)
    if kind in ('solve', 'serve'):
        if kind == 'solve':
            sizes, m, it, s = [case['nxy'] ** 2 * case['nz']], case['m'], case['iters'], 16
        else:
            sizes = [2 * a * a * b for a, b in SWEEP[:case['dots']]]
            m, it = case['k'] + max(2, case['k'] // 2), case['ticks']
            s = 16 if case['phase'] == 'c128' else 8
        n = 8 * sum(sizes)
        # an iteration reads X, AX, P, AP and writes them, applies H twice to the residual, forms
        # [X R P]^H [AR AP] and the two-output Ritz updates
        return dict(bytes=float(it) * n * m * s * 12,
                    flops=float(it) * n * m * (4 * _FMA[8] / 8 + 8.0 * m * (6 + 5)))
    if kind == 'ritz':
        n, m = case['n'], case['m']
        s = 16 if case['dtype'] == 'c128' else 8
        return dict(bytes=float(n) * m * s * (3 + 2 + 3 + 1), flops=8.0 * n * m * m * (6 + 3))
    N = case['nxy'] ** 2 * case['nz']
    # about twelve conjugate-gradient steps: stencil, two transforms of three components, updates
    return dict(bytes=12.0 * N * 3 * 8 * 10, flops=12.0 * N * (27 * 18 + 2 * 3 * 2.5 * math.log2(N)))


# --------------------------------------------------------------------------------------------
# Results in 64 bits
# --------------------------------------------------------------------------------------------

class _Pryor:
    """Pryor's eight-band table on a hard-walled grid, applied term by term in complex128."""

    def __init__(self, f, shape, h, bands):
        self.shape, self.h, self.bands = shape, h, bands
        self.f = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda().double()[..., None]
                  for k, v in f.items()}

    def shift(self, x, axis, d):
        """x at the neighbour in direction d along axis, zero beyond the wall."""
        y = torch.zeros_like(x)
        n = x.shape[axis]
        if n > 1:
            y.narrow(axis, 0 if d > 0 else 1, n - 1).copy_(x.narrow(axis, 1 if d > 0 else 0, n - 1))
        return y

    def D(self, a, x):
        return (-1j / (2 * self.h)) * (self.shift(x, a, 1) - self.shift(x, a, -1))

    def k2(self, al, a, x):
        out = torch.zeros_like(x)
        n = x.shape[a]
        for d in (1, -1):
            t = 0.5 * (al + self.shift(al, a, d))
            wall = n - 1 if d > 0 else 0
            t.narrow(a, wall, 1).copy_(al.narrow(a, wall, 1))
            out += t * (x - self.shift(x, a, d))
        return out / self.h ** 2

    def cross(self, al, a, b, x):
        return 0.5 * (self.D(a, al * self.D(b, x)) + self.D(b, al * self.D(a, x)))

    def sym(self, c, a, x):
        return 0.5 * (c * self.D(a, x) + self.D(a, c * x))

    def apply(self, X):
        f, m = self.f, X.shape[1]
        lo = 0 if self.bands == 8 else 2
        xs = X.reshape((self.bands,) + self.shape + (m,))
        zero = torch.zeros_like(xs[0])
        x = [xs[b - lo] if lo <= b < lo + self.bands else zero for b in range(8)]
        s2, s3, s6, s32 = (math.sqrt(v) for v in (2.0, 3.0, 6.0, 1.5))
        g1, g2, g3, P0 = f['gamma1'], f['gamma2'], f['gamma3'], f['P0']
        ones = torch.ones_like(g1)
        qe = -(f['b'] / 2) * (f['exx'] + f['eyy'] - 2 * f['ezz'])
        re = s3 / 2 * f['b'] * (f['exx'] - f['eyy']) - 1j * f['d'] * f['exy']
        se = -f['d'] * (f['ezx'] - 1j * f['eyz'])

        def A(v):
            return f['Ec'] * v + G * sum(self.k2(ones, a, v) for a in range(3))

        def P(v):
            return -f['Ev'] * v + G * sum(self.k2(g1, a, v) for a in range(3))

        def Q(v):
            return qe * v + G * (self.k2(g2, 0, v) + self.k2(g2, 1, v) - 2 * self.k2(g2, 2, v))

        def R(v, c=1):
            w = re if c > 0 else re.conj()
            return w * v + G * (-s3 * (self.k2(g2, 0, v) - self.k2(g2, 1, v))
                                + c * 2j * s3 * self.cross(g3, 0, 1, v))

        def S(v, c=1):
            w = se if c > 0 else se.conj()
            return w * v + 2 * s3 * G * (self.cross(g3, 2, 0, v) - c * 1j * self.cross(g3, 2, 1, v))

        def U(v):
            return (self.sym(P0 * (1 - f['ezz']), 2, v) - self.sym(P0 * f['ezx'], 0, v)
                    - self.sym(P0 * f['eyz'], 1, v)) / s3

        def V(v, c=1):
            i = c * 1j
            return (self.sym(P0, 0, v) - i * self.sym(P0, 1, v)
                    - self.sym(P0 * f['exx'], 0, v) + i * self.sym(P0 * f['exy'], 0, v)
                    - self.sym(P0 * f['exy'], 1, v) + i * self.sym(P0 * f['eyy'], 1, v)
                    - self.sym(P0 * f['ezx'], 2, v) + i * self.sym(P0 * f['eyz'], 2, v)) / s6

        def Rh(v):
            return R(v, -1)

        def Sh(v):
            return S(v, -1)

        def Vh(v):
            return V(v, -1)
        y = [torch.zeros_like(zero) for _ in range(8)]
        Dl = f['delta_so']
        for b in range(2):
            if self.bands == 8:
                y[b] += A(x[b])
        for b in range(2, 8):
            y[b] += -P(x[b]) - (Dl * x[b] if b > 5 else 0.0)
        for b, sg in ((2, 1), (3, -1), (4, -1), (5, 1)):
            y[b] += sg * Q(x[b])
        y[2] += -Sh(x[3]) + R(x[4]) + s32 * S(x[6]) - s2 * Q(x[7])
        y[3] += -S(x[2]) + R(x[5]) - s2 * R(x[6]) + S(x[7]) / s2
        y[4] += Rh(x[2]) + Sh(x[5]) + Sh(x[6]) / s2 + s2 * Rh(x[7])
        y[5] += Rh(x[3]) + S(x[4]) + s2 * Q(x[6]) + s32 * Sh(x[7])
        y[6] += s32 * Sh(x[2]) - s2 * Rh(x[3]) + S(x[4]) / s2 + s2 * Q(x[5])
        y[7] += -s2 * Q(x[2]) + Sh(x[3]) / s2 + s2 * R(x[4]) + s32 * S(x[5])
        if self.bands == 8:
            y[0] += Vh(x[2]) + s3 * V(x[4]) - s2 * U(x[5]) - U(x[6]) + s2 * Vh(x[7])
            y[1] += -s2 * U(x[2]) - s3 * Vh(x[3]) - V(x[5]) + s2 * V(x[6]) + U(x[7])
            y[2] += V(x[0]) - s2 * U(x[1])
            y[3] += -s3 * V(x[1])
            y[4] += s3 * Vh(x[0])
            y[5] += -s2 * U(x[0]) - Vh(x[1])
            y[6] += -U(x[0]) + s2 * Vh(x[1])
            y[7] += s2 * V(x[0]) + U(x[1])
        out = torch.stack(y[lo:lo + self.bands]).reshape(X.shape)
        return out if self.bands == 8 else -out          # hole convention


def exact(case, seed):
    if case['kind'] == 'apply':
        f, se, _ = _environment(case['nxy'], case['nz'], case['h'], case['bands'], seed)
        op = _Pryor(f, (case['nxy'], case['nxy'], case['nz']), case['h'], case['bands'])
        dt = torch.complex128 if case['dtype'] == 'c128' else torch.complex64
        X = _block(case['bands'] * case['nxy'] ** 2 * case['nz'], case['m'], seed, dt)
        Y = torch.empty(X.shape, dtype=torch.complex128, device='cuda')
        for c in range(0, case['m'], 4):
            x = X[:, c:c + 4].to(torch.complex128)
            y = op.apply(x)
            if case['mode'] != 'plain':
                y = y - se * x
            if case['mode'] == 'folded':
                y = op.apply(y) - se * y
            Y[:, c:c + 4] = y
        return Y
    if case['kind'] == 'ritz':
        W, A, C = _ritz_inputs(case, seed)
        W, A = W.to(torch.complex128), A.to(torch.complex128)
        return dict(gram=W.conj().T @ A, update=W @ torch.from_numpy(C).cuda())
    # the iterations (solve, serve, strain) have no value of their own beside their iterates
    return None
