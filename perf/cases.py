"""The work this package is used for, as cases that can be timed and compared.

A case is one pass through a public entry point, with the sizes, networks and
precisions its users run:

* ``step``     the drop-in step of the reference's loop (``Ros2GPU.solver``):
               one column's arrays uploaded, one Ros2 attempt, results read back.
* ``attempt``  one attempt of a batch that stays loaded: new states in, results out.
* ``profile``  the same after the atmosphere changed (a retrieval, a T-P sweep):
               rate constants recomputed on the device, then the attempt.
* ``run``      the batched loop: Ros2 steps with step control on the device.
* ``photo``    a radiative-transfer update of a batch before its next steps.
* ``mlp``      one layer of the learned start's training step, forward and backward.
* ``solve``    the block-tridiagonal solve on buffers the caller owns.

States are seeded: profiles and mixing ratios near this package's recorded
steady states (tests/golden), as a learned start or a restart gives them, or the
constant-mixing start (``run``, and the networks without recorded states).
"""
import ctypes
import math
import os

import numpy as np
import torch

from vulcan_gb300 import batch, capi, column, configs, photo
from vulcan_gb300.network import Network
from vulcan_gb300.solver import ColumnBatch, GPUNetwork, Ros2Handle, ctrl_from

GOLDEN = os.path.join('tests', 'golden')
NETS = {'CHO': 'net_CHO_thermo.npz', 'NCHO': 'net_NCHO_thermo.npz',
        'NCHO_photo': 'net_NCHO_photo.npz', 'SNCHO': 'net_SNCHO_photo.npz',
        'SYN150': 'net_SYN150_photo.npz'}
# species, reaction pairs and Jacobian entries of a diagonal block
SIZES = {'CHO': (41, 207), 'NCHO': (69, 391), 'NCHO_photo': (69, 439), 'SNCHO': (89, 575),
         'SYN150': (150, 1261)}
MAX_PROFILES = 32           # distinct T-P-Kzz profiles of a batch; its states all differ
R_ROS = 1. + 1. / 2. ** 0.5
KB, NAVO = 1.38064852E-16, 6.02214086E+23
HC = 1.98644582E-9

_nets = {}


def _net(name):
    if name not in _nets:
        _nets[name] = Network.from_npz(os.path.join(GOLDEN, NETS[name]))
    return _nets[name]


def _atoms(name):
    a = ['H', 'O', 'C', 'He']
    return a if name == 'CHO' else a + ['N', 'S'] if name == 'SNCHO' else a + ['N']


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: config 0's single CHO column inside the reference's own loop
        dict(name='step_cho', kind='step', net='CHO', ncols=1, nz_lo=100, nz_hi=100,
             precision='fp64', log_dt=-6.0),
        # the same for a photochemical column (config 1), the usual single-planet run
        dict(name='step_ncho_photo', kind='step', net='NCHO_photo', ncols=1, nz_lo=150, nz_hi=150,
             precision='fp64', log_dt=-7.5),
        # a few columns of the sulfur network (hot-Jupiter grids), uneven and odd sizes
        dict(name='attempt_sncho_7', kind='attempt', net='SNCHO', ncols=7, nz_lo=61, nz_hi=149,
             precision='fp64', log_dt=-6.0),
        # an ensemble of uneven columns, full precision
        dict(name='attempt_ncho_64', kind='attempt', net='NCHO', ncols=64, nz_lo=60, nz_hi=200,
             precision='fp64', log_dt=-7.0),
        # the ensemble after new temperature profiles, mixed precision
        dict(name='profile_ncho_96', kind='profile', net='NCHO', ncols=96, nz_lo=60, nz_hi=200,
             precision='mixed', log_dt=-7.5),
        # the headline batch: 512 uneven columns, mixed and plain FP64
        dict(name='run_ncho_512_mixed', kind='run', net='NCHO', ncols=512, nz_lo=60, nz_hi=200,
             precision='mixed', steps=3),
        dict(name='run_ncho_512_fp64', kind='run', net='NCHO', ncols=512, nz_lo=60, nz_hi=200,
             precision='fp64', steps=2),
        # the large-network stress workload (150 species, nz = 200)
        dict(name='attempt_syn150_48', kind='attempt', net='SYN150', ncols=48, nz_lo=200, nz_hi=200,
             precision='mixed', log_dt=-6.0),
        # radiative transfer of a batch: 446 wavelength bins, 48 photolysis channels
        dict(name='photo_128', kind='photo', net='NCHO_photo', ncols=128, nz_lo=150, nz_hi=150),
        # a hidden layer of the learned start's network at its training batch size
        dict(name='mlp_hidden', kind='mlp', rows=4096, width_in=512, width_out=512),
        # its first layer (92 features) on one column's layers: ragged sizes
        dict(name='mlp_small', kind='mlp', rows=150, width_in=92, width_out=512),
        # a caller's own block-tridiagonal system, nothing allocated
        dict(name='solve_69', kind='solve', species=69, layers=150),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['step', 'attempt', 'attempt', 'profile', 'run', 'run', 'photo', 'mlp', 'solve'])
    precision = rng.choice(['fp64', 'mixed'])
    if kind == 'mlp':
        return dict(kind='mlp', rows=_log(rng, 60, 4096), width_in=rng.choice([92, 512, rng.randint(23, 512)]),
                    width_out=rng.choice([512, 69, rng.randint(41, 512)]))
    if kind == 'solve':
        ni = rng.randint(20, 99)
        return dict(kind='solve', species=ni, layers=rng.randint(20, min(200, (1 << 21) // (ni * (ni + 1)) - 1)))
    if kind == 'photo':
        return dict(kind='photo', net='NCHO_photo', ncols=_log(rng, 1, 128), nz_lo=60, nz_hi=rng.randint(60, 150))
    if kind == 'run':
        return dict(kind='run', net=rng.choice(['CHO', 'NCHO', 'NCHO']), ncols=_log(rng, 4, 512), nz_lo=60,
                    nz_hi=rng.randint(90, 200), precision=precision, steps=rng.randint(1, 2))
    net = rng.choice(['CHO', 'NCHO', 'NCHO_photo', 'SNCHO', 'SYN150'])
    if net == 'SNCHO':
        precision = 'fp64'
    if net in ('SNCHO', 'SYN150'):
        log_dt = rng.uniform(-6.3, -5.8)
    else:
        log_dt = rng.uniform(-8.5, -7.) if precision == 'mixed' else rng.uniform(-8., -6.)
    nz = rng.randint(60, 200)
    if kind == 'step':
        return dict(kind='step', net=net, ncols=1, nz_lo=nz, nz_hi=nz, precision=precision, log_dt=log_dt)
    most = 48 if net == 'SYN150' else 128
    return dict(kind=kind, net=net, ncols=_log(rng, 2, most), nz_lo=60, nz_hi=nz,
                precision=precision, log_dt=log_dt)


# ------------------------------------------------------------ inputs from a seed
_steady = []


def _recorded():
    """This package's recorded steady states (tests/golden), NCHO species: for
    each column its log10 P (bar), T, log10 Kzz and log10 mixing ratios."""
    if not _steady:
        d = np.load(os.path.join(GOLDEN, 'warmstart_holdout.npz'))
        for c in np.unique(d['col']):
            r = np.flatnonzero(d['col'] == c)
            r = r[np.argsort(d['X'][r, 0])]
            X, Y = d['X'][r].astype(float), d['Y'][r].astype(float)
            _steady.append((X[:, 0], 1000. * X[:, 1], X[0, 2], Y))
    return _steady


def _sizes(case):
    """Layer counts of the case's columns: the same for every seed."""
    n = min(case['ncols'], MAX_PROFILES)
    rng = np.random.default_rng(97 * case['ncols'] + case['nz_hi'])
    nz = rng.integers(case['nz_lo'], case['nz_hi'] + 1, n)
    return [int(nz[c % n]) for c in range(case['ncols'])]


def _specs(case, rng):
    """Seeded column specifications (configs.ColumnSpec): temperatures within
    2 % of a recorded profile, abundances as configs.config2_columns."""
    net = _net(case['net'])
    out = []
    for nz in _sizes(case)[:MAX_PROFILES]:
        pco = configs.log_p_grid(nz)
        which = int(rng.integers(len(_recorded())))
        logp, T, logK, _ = _recorded()[which]
        T = np.interp(np.log10(pco / 1e6), logp, T) * (1. + rng.uniform(-0.02, 0.02))
        mix = configs.solar_mix(met=10. ** rng.uniform(-1., 2.), c_to_o=rng.uniform(0.3, 1.2),
                                with_n=case['net'] != 'CHO')
        if case['net'] == 'SNCHO':
            mix['H2S'] = 2.2e-5
        J = None
        if net.use_photo:
            J = configs.photo_J_profile(rng, pco, sorted(net.photo_index()))
        spec = configs.ColumnSpec(network=NETS[case['net']], use_photo=net.use_photo, pco=pco, Tco=T,
                                  Kzz=np.full(nz - 1, 10. ** (logK + rng.uniform(-0.5, 0.5))), const_mix=mix,
                                  atom_list=_atoms(case['net']), conver_ignore=[], photo_J=J)
        out.append((spec, which))
    return out


def _near_steady(net, pco, which, rng):
    """Mixing ratios of a recorded steady state on the grid, each within some
    5 % of it: what a learned start or a restart hands to the solver.  A
    species below 1e-12 starts absent, as the constant-mixing start leaves it."""
    logp, _, _, x = _recorded()[which]
    names = {s: i for i, s in enumerate(_net('NCHO').species)}
    g = np.log10(pco / 1e6)
    x = np.stack([np.interp(g, logp, x[:, names[s]]) for s in net.species], axis=1)
    return np.where(x > -12., 10. ** (x + 0.02 * rng.standard_normal(x.shape)), 0.)


def _columns(case, seed):
    """(network, items): what batch.build_items gives for the case's columns,
    each with a state of its own."""
    rng = np.random.default_rng(seed)
    net = _net(case['net'])
    specs = _specs(case, rng)
    base = batch.build_items([sp for sp, _ in specs], net)
    known = set(net.species) <= set(_net('NCHO').species)
    items = []
    for c in range(case['ncols']):
        it = dict(base[c % len(base)])
        col = it['col']
        if case['kind'] == 'run' or not known:   # the constant-mixing start, its abundances varied
            y = it['y'] * np.exp(0.05 * rng.standard_normal(net.ni))
        else:
            y = _near_steady(net, col.pco, specs[c % len(base)][1], rng)
            y *= (col.n_0 / y.sum(axis=1))[:, None]
        it['y'], it['ymix'] = y, y / y.sum(axis=1, keepdims=True)
        it['atom_ini'] = column.atom_totals(net, y, _atoms(case['net']))
        items.append(it)
    return net, items


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _tables():
    """The wavelength tables of the photochemical column (tests/golden)."""
    return photo.PhotoTables.from_fixture(np.load(os.path.join(GOLDEN, 'golden_c1rt.npz')))


def _mlp_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    B, K, N = case['rows'], case['width_in'], case['width_out']
    r = lambda *s: torch.randn(*s, generator=g)
    X = torch.nn.functional.silu(r(B, K)).to(torch.bfloat16)
    W = (r(K, N) * K ** -0.5).to(torch.bfloat16)
    b = 0.1 * r(N)
    Z = (X.float() @ W.float() + b + 0.01 * r(B, N))     # kept from an earlier forward pass
    dH = r(B, N) * (2.0 / (B * N))
    return X, W, b, Z, dH


def _solve_inputs(case, seed):
    """A system like a Ros2 step's: 1/dt plus the loss rates on the diagonal,
    sparse production terms, diffusion between layers."""
    rng = np.random.default_rng(seed)
    nz, n = case['layers'], case['species']
    P = rng.random((nz, n, n)) * (rng.random((nz, n, n)) < 0.3) * 10. ** rng.uniform(-4., 0., (nz, n, n))
    D = -P
    i = np.arange(n)
    lo, up = rng.random((nz, n)), rng.random((nz, n))
    D[:, i, i] = P.sum(axis=1) + lo + up + 10. ** rng.uniform(-1., 1., (nz, n))
    return D, -lo, -up, rng.standard_normal((nz, n))


def prepare(case, seed):
    kind = case['kind']
    if kind == 'mlp':
        X, W, b, Z, dH = (t.cuda().contiguous() for t in _mlp_inputs(case, seed))
        return dict(kind=kind, X=X, W=W, b=b, Z=Z, dH=dH)
    if kind == 'solve':
        t = [torch.from_numpy(a).cuda() for a in _solve_inputs(case, seed)]
        return dict(kind=kind, t=t, x=torch.empty_like(t[3]))
    net, items = _columns(case, seed)
    b = ColumnBatch(items, net.ni)
    precision = capi.VK_PREC_MIXED if case.get('precision') == 'mixed' else capi.VK_PREC_FP64
    h = Ros2Handle(GPUNetwork(net, _atoms(case['net'])), b.ncols, b.L, precision)
    s = dict(kind=kind, h=h, batch=b, items=items, ni=net.ni)
    if kind != 'step':
        h.set_columns(b)
        s['y'], s['ymix'] = _pinned(b.y), _pinned(b.ymix)
    if kind == 'photo':
        photo.attach(h, _tables(), net)
    elif kind == 'run':
        h.set_atom_ini(np.stack([it['atom_ini'] for it in items]))
        s['ctrl'] = ctrl_from(None, gs=configs.GS, Rp=configs.RP)
        s['steps'] = case['steps']
        s['out'] = {k: _pinned(np.empty(n, dtype=t)) for k, n, t in
                    [(k, (b.L, net.ni), np.float64) for k in ('y', 'ymix')]
                    + [(k, b.ncols, np.float64) for k in ('dt', 't', 'delta')]
                    + [(k, b.ncols, np.int32) for k in ('count', 'end_case')]}
    else:
        s['dt'] = 10. ** case['log_dt']
    if kind == 'profile':
        h.set_rate_params(net)
    return s


# --------------------------------------------------------------------- one pass
def run(state):
    kind = state['kind']
    if kind == 'mlp':
        return _run_mlp(state)
    if kind == 'solve':
        p = [ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))
             for t in state['t'] + [state['x']]]
        nz, n = state['x'].shape
        capi.check(capi.lib().vk_block_solve_noalloc(nz, n, *p, None))
        return state['x']
    h = state['h']
    if kind == 'step':                       # as Ros2GPUMixin.solver does it
        h.set_columns(ColumnBatch(state['items'], state['ni']))
        return h.attempt(state['dt'])
    if kind == 'photo':
        capi.check(capi.lib().vk_photo_reset(h.h), h.h)
        change = h.photo_update()
        J = np.empty((state['batch'].L, h.photo_dims[1]))
        capi.check(capi.lib().vk_photo_get(h.h, None, None, capi.ptr(J)), h.h)
        return dict(change=change, J=J)
    h.set_state(state['y'], state['ymix'])
    if kind == 'run':
        h.set_clock(dt=1e-10, t=0.0, count=1)
        h.run(state['ctrl'], max_steps=state['steps'])
        return h.state(state['out'])
    if kind == 'profile':
        h.set_atm(state['batch'].atm)
        h.compute_k()
    return h.attempt(state['dt'])


def _run_mlp(s):
    L = capi.lib()
    X, W = s['X'], s['W']
    B, K, N = X.shape[0], X.shape[1], W.shape[1]
    new = lambda *shape, dtype=torch.float32: torch.empty(*shape, device=X.device, dtype=dtype)
    v = lambda t: ctypes.c_void_p(t.data_ptr())
    f = lambda t: ctypes.cast(v(t), ctypes.POINTER(ctypes.c_float))
    Z, H = new(B, N), new(B, N, dtype=torch.bfloat16)
    capi.check(L.vk_mlp_forward(B, K, N, v(X), v(W), f(s['b']), f(Z), v(H), 1, None))
    dZ, dW, db, dX = new(B, N, dtype=torch.bfloat16), new(K, N), new(N), new(B, K)
    capi.check(L.vk_mlp_backward(B, K, N, v(X), v(W), f(s['Z']), f(s['dH']), 1, v(dZ), f(dW), f(db),
                                 f(dX), None))
    return dict(Z=Z, H=H, dZ=dZ, dW=dW, db=db, dX=dX)


# ------------------------------------------------------------------------- work
def work(case):
    kind = case['kind']
    if kind == 'mlp':
        B, K, N = case['rows'], case['width_in'], case['width_out']
        return dict(bytes=2 * (B * K + K * N + 2 * B * N) + 4 * (N + 3 * B * N + K * N + N + B * K),
                    flops=6 * B * K * N)
    if kind == 'solve':
        nz, n = case['layers'], case['species']
        return dict(bytes=8 * nz * (n * n + 4 * n), flops=nz * (2 * n ** 3 + 4 * n * n))
    ni, npair = SIZES[case['net']]
    L = case['ncols'] * (case['nz_lo'] + case['nz_hi']) / 2
    if kind == 'photo':
        nb, nch, nab = 446, 48, 29
        return dict(bytes=L * 8 * (2 * ni + 4 * nb + nch), flops=L * nb * (3 * nab + 2 * nch + 120))
    # the rate constants, the state in and out, the atmosphere; the block
    # inverses and their products with four right-hand sides
    one = dict(bytes=L * 8 * (2 * npair + 4 * ni + ni + capi.ATM_NF),
               flops=L * (2 * ni ** 3 + 8 * ni * ni + 20 * npair))
    n = case.get('steps', 1)
    return {k: v * n for k, v in one.items()}


# ------------------------------------------------------------ the values in 64 bits
def exact(case, seed):
    """What run() returns for the same inputs, in plain 64-bit torch and numpy
    (the set-up arrays are inputs).  None for the batched loop: hundreds of
    dense blocks a layer and attempt take longer than a case may."""
    kind = case['kind']
    if kind == 'mlp':
        X, W, b, Z0, dH = (t.double() for t in _mlp_inputs(case, seed))
        Z = X @ W + b
        sg = torch.sigmoid(Z0)
        dZ = dH * (sg * (1. + Z0 * (1. - sg)))
        dZb = dZ.float().to(torch.bfloat16).double()    # the gradients take the rounded one
        return dict(Z=Z, H=torch.nn.functional.silu(Z), dZ=dZ, dW=X.T @ dZb, db=dZb.sum(0), dX=dZb @ W.T)
    if kind == 'solve':
        D, lo, up, b = (torch.from_numpy(a) for a in _solve_inputs(case, seed))
        return _block_solve(D[:, None], lo[:, None], up[:, None], [b.shape[0]], b[:, None])[:, 0]
    if kind == 'run':
        return None
    net, items = _columns(case, seed)
    if kind == 'photo':
        return _exact_photo(net, items)
    return _exact_attempt(net, items, 10. ** case['log_dt'])


def _block_solve(D, lo, up, nzs, *rhs):
    """Block-Thomas with pivoted LU of every block; D [nz][columns][n][n], the
    columns in decreasing order of their layer counts nzs."""
    nz, ncols = D.shape[:2]
    alive = [sum(1 for z in nzs if z > j) for j in range(nz)]
    Gs, out = [], []
    for j in range(nz):
        m = alive[j]
        A = D[j, :m].clone()
        if j:
            A -= lo[j, :m, :, None] * Gs[-1][:m] * up[j - 1, :m, None, :]
        Gs.append(torch.linalg.inv(A))
    for b in rhs:
        z, x = [], torch.zeros_like(b)
        for j in range(nz):
            v = b[j, :alive[j]] - (lo[j, :alive[j]] * z[-1][:alive[j]] if j else 0.)
            z.append((Gs[j] @ v[..., None])[..., 0])
        for j in range(nz - 1, -1, -1):
            m = alive[j]
            x[j, :m] = z[j]
            if j + 1 < nz and alive[j + 1]:
                k = alive[j + 1]
                x[j, :k] -= (Gs[j][:k] @ (up[j, :k] * x[j + 1, :k])[..., None])[..., 0]
        out.append(x)
    return out[0] if len(out) == 1 else out


def _sides(net):
    s = {name: i for i, name in enumerate(net.species)}
    return [[[(nu, -1 if name == 'M' else s[name]) for nu, name in side] for side in (r.reac, r.prod)]
            for r in net.reactions]


def _product(terms, y, M, skip=None):
    """k-free mass action of one side; its derivative by species `skip`."""
    e, v = {}, None
    for nu, s in terms:
        e[s] = e.get(s, 0) + nu
    for s, nu in e.items():
        f = M if s < 0 else y[s]
        if s == skip:
            f = nu * f ** (nu - 1) if nu > 1 else None
        elif nu != 1:
            f = f ** nu
        if f is not None:
            v = f if v is None else v * f
    return torch.ones_like(M) if v is None else v


def _exact_attempt(net, items, dt):
    order = sorted(range(len(items)), key=lambda c: -items[c]['col'].nz)
    nzs = [items[c]['col'].nz for c in order]
    nz, nc, n = nzs[0], len(items), net.ni
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'

    def pack(get, width=()):                  # [nz][columns]..., padded with ones
        a = np.ones((nz, nc) + width)
        for i, c in enumerate(order):
            v = get(items[c])
            a[:v.shape[0], i] = v
        return torch.from_numpy(a).to(dev)

    y0 = pack(lambda it: it['y'], (n,))
    ymix = pack(lambda it: it['ymix'], (n,))
    k = pack(lambda it: it['k'].T, (net.nr,))
    M = pack(lambda it: it['col'].M)
    sides = _sides(net)
    last = torch.tensor([z - 1 for z in nzs], device=dev)
    jj = torch.arange(nz, device=dev)[:, None]
    inside, top = jj <= last, jj == last
    # transport: the flux through the interface above layer j is
    #   K+D over dz times the mixing-ratio difference of the mean density, plus the drift
    dzi = pack(lambda it: it['col'].dzi)
    Dz = pack(lambda it: it['col'].Dzz, (n,))
    Kz = pack(lambda it: it['col'].Kzz)
    Ti, Hpi = pack(lambda it: it['col'].Ti), pack(lambda it: it['col'].Hpi)
    T, g = pack(lambda it: it['col'].Tco), pack(lambda it: it['col'].g)
    ms = torch.from_numpy(items[0]['col'].ms).to(dev)
    al = torch.from_numpy(items[0]['col'].alpha).to(dev)
    up_ok = (jj < last).double()[..., None]
    shift = lambda a: torch.cat([a[1:], a[-1:]])          # layer j + 1
    back = lambda a: torch.cat([a[:1], a[:-1]])           # layer j - 1
    dn_ok = back(up_ok).clone()
    dn_ok[0] = 0.
    dTdz = (shift(T) - T) / dzi

    def phi(gr):
        return -1. / Hpi[..., None] + ms * gr[..., None] / (NAVO * KB * Ti[..., None]) \
            + (dTdz / Ti)[..., None] * al

    da = torch.where(jj == 0, dzi, 0.5 * (back(dzi) + dzi))
    da = torch.where(top, back(dzi), da)[..., None]
    # the drift takes the gravity of the layer whose density it carries, but
    # an end layer's own on both sides
    g_up = torch.where(jj == 0, g, shift(g))
    g_dn = torch.where(top, g, back(g))

    def transport(y):
        ys = y.sum(-1)
        mean_u, mean_d = (shift(ys) + ys) / 2., (ys + back(ys)) / 2.
        KD = Kz[..., None] + Dz
        KDm = back(KD)
        dm = back(dzi)[..., None]
        gu, gd = KD / dzi[..., None] / da * up_ok, KDm / dm / da * dn_ok
        hu, hd = Dz / (2. * da) * up_ok, back(Dz) / (2. * da) * dn_ok
        A = -gu * (mean_u / ys)[..., None] - gd * (mean_d / ys)[..., None] + hu * phi(g) \
            - hd * back_phi(g)
        B = gu * (mean_u / shift(ys))[..., None] + hu * phi(g_up)
        Cc = gd * (mean_d / back(ys))[..., None] - hd * back_phi(g_dn)
        return A, B, Cc

    def back_phi(gr):                         # phi of the interface below, gravity gr of this layer
        return -1. / back(Hpi)[..., None] + ms * gr[..., None] / (NAVO * KB * back(Ti)[..., None]) \
            + back(dTdz / Ti)[..., None] * al

    def rhs(y):
        f = torch.zeros_like(y)
        ysp = y.unbind(-1)
        for p, (reac, prod) in enumerate(sides):
            v = k[..., 2 * p] * _product(reac, ysp, M) - k[..., 2 * p + 1] * _product(prod, ysp, M)
            for sign, side in ((-1., reac), (1., prod)):
                for nu, s in side:
                    if s >= 0:
                        f[..., s] += sign * nu * v
        A, B, Cc = transport(y)
        return f + A * y + B * shift(y) + Cc * back(y), A, B, Cc

    f1, A, B, Cc = rhs(y0)
    D = torch.zeros(nz, nc, n, n, dtype=torch.float64, device=dev)
    ysp = y0.unbind(-1)
    for p, two in enumerate(sides):
        net_nu = {}
        for sign, side in ((-1, two[0]), (1, two[1])):
            for nu, s in side:
                if s >= 0:
                    net_nu[s] = net_nu.get(s, 0) + sign * nu
        for q in {s for side in two for _, s in side if s >= 0}:
            d = 0.
            for w, side in enumerate(two):
                if any(s == q for _, s in side):
                    d = d + (1. - 2. * w) * k[..., 2 * p + w] * _product(side, ysp, M, skip=q)
            for s, nu in net_nu.items():
                if nu:
                    D[..., s, q] -= nu * d
    i = torch.arange(n, device=dev)
    D[..., i, i] += 1. / (R_ROS * dt) - A
    k1 = _block_solve(D, -Cc, -B, nzs, f1)
    yk2 = y0 + k1 / R_ROS
    f2 = rhs(yk2)[0] - 2. / (R_ROS * dt) * k1
    k2 = _block_solve(D, -Cc, -B, nzs, f2)
    sol = y0 + 1.5 / R_ROS * k1 + 0.5 / R_ROS * k2
    d = (sol - yk2).abs()
    d[(ymix < 1e-22) | (sol < 0.1)] = 0.
    ratio = torch.where((sol > 0) & inside[..., None], d / sol, torch.zeros_like(d))
    delta = ratio.amax(dim=(0, 2))
    ym = sol / sol.sum(-1, keepdim=True)
    place = [order.index(c) for c in range(nc)]
    cat = lambda a: torch.cat([a[:nzs[i], i] for i in place]).cpu()
    return dict(sol=cat(sol), ymix=cat(ym), delta=delta[place].cpu())


def _exact_photo(net, items):
    """tau, the two-stream fluxes from zero diffuse flux, and J (op.py:2580-2786)."""
    t = _tables()
    sp = {s: i for i, s in enumerate(net.species)}
    w = t.weights()
    J, change = [], []
    cosz, edd = math.cos(t.sl_angle), t.edd
    mu = -cosz
    ab, sc = [sp[s] for s in t.absp_sp], [sp[s] for s in t.scat_sp]
    for it in items:
        y, ymix, col = it['y'], it['ymix'], it['col']
        nz = col.nz
        dtau = (y[:, ab] * col.dz[:, None]) @ t.cross + (y[:, sc] * col.dz[:, None]) @ t.cross_scat
        tau = np.concatenate([np.cumsum(dtau[::-1], axis=0)[::-1], np.zeros((1, len(t.bins)))])
        tot = ymix[:, ab] @ t.cross
        sca = ymix[:, sc] @ t.cross_scat
        with np.errstate(divide='ignore', invalid='ignore'):
            w0 = np.minimum(np.nan_to_num(sca / (tot + sca)), 1. - 1.e-8)
        sq = np.sqrt(1. - w0)
        tran = np.exp(-sq * (tau[:-1] - tau[1:]) / edd)
        zp, zm = 0.5 * (1. + sq), 0.5 * (1. - sq)
        ll = -w0 / (1. / mu ** 2 - (1. - w0) / edd ** 2)
        gp, gm = 0.5 * ll * (1. / edd + 1. / mu), 0.5 * ll * (1. / edd - 1. / mu)
        chi, xi, ph = zm ** 2 * tran ** 2 - zp ** 2, zp * zm * (1. - tran ** 2), (zm ** 2 - zp ** 2) * tran
        s = t.sflux_top * np.exp(-tau / cosz)
        d = s * cosz
        iu = ph * gp * d[:-1] - (xi * gm + chi * gp) * d[1:]
        idn = ph * gm * d[1:] - (chi * gm + xi * gp) * d[:-1]
        dd, du = np.zeros_like(tau), np.zeros_like(tau)
        for j in range(nz - 1, -1, -1):
            dd[j] = (ph[j] * dd[j + 1] + idn[j] / mu) / chi[j]
        for j in range(1, nz + 1):
            du[j] = (ph[j - 1] * du[j - 1] - xi[j - 1] * dd[j] + iu[j - 1] / mu) / chi[j - 1]
        af = (0.5 * (s[:-1] + s[1:]) + 0.5 * (du[:-1] + du[1:] + dd[1:] + dd[:-1]) / edd) / (HC / t.bins)
        J.append(af @ (t.cross_J * w).T)
        change.append(1.0 if (af > t.flux_atol).any() else 0.0)     # from zero flux
    return dict(change=np.array(change), J=np.concatenate(J))
