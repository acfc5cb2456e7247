"""The engine's timed cases: the calls a user of this framework makes, through
its public entry points, from one water to the largest molecules whose build
takes under two seconds.

A case is a dict of plain values:
  op        jk (direct J/K build), energy (E2 and its gradient by autograd),
            gradjk (gradient J/K), fill (s8 integral tensor), incore (J/K from
            a stored tensor), batch (J/K of many molecules)
  mol       water (clusters on a cubic lattice) or alkane; n the number of
            waters or carbons (batch: the number of molecules, each of 1 to 16
            waters); basis 631g, dz or tz
  n_dm, hermi, precision ('fp64', 'mixed'), side ('host', 'device'), delta (a
            late-SCF density change), sym ('s8', 's4') and nao where they apply
Geometries, densities and stored tensors are drawn from the seed.
"""
import math

import numpy
import torch

from pyscf_b200 import _vhf, flops, grad, incore, lib

BOHR = 0.52917721092

# (l, exponents, contraction columns) of every shell, radially normalised
# as PySCF keeps them in env
BASIS = {
    '631g': {
        8: [(0, [5484.6717, 825.23495, 188.04696, 52.9645, 16.89757, 5.7996353],
             [[2.94842454771, 5.42657123619, 8.78126489322, 11.543212924, 9.90055015194, 3.38516599422]]),
            (0, [15.539616, 3.5999336, 1.0137618], [[-2.19051792395, -0.977405527727, 2.88629094359]]),
            (0, [0.2700058], [[0.946334872683]]),
            (1, [15.539616, 3.5999336, 1.0137618], [[6.37930733662, 4.91490974732, 2.15791054616]]),
            (1, [0.2700058], [[0.56780702218]])],
        1: [(0, [18.731137, 2.8253937, 0.6401217], [[0.761926219817, 1.2923709967, 1.47131900254]]),
            (0, [0.1612778], [[0.642977783424]])]},
    'dz': {
        8: [(0, [11720.0, 1759.0, 400.8, 113.7, 37.03, 13.27, 5.025, 1.013],
             [[2.01953999996, 3.75176051046, 6.29675239515, 9.21467522873, 10.7298896828, 7.87818279244,
               2.29637501267, 0.0394147511498],
              [-0.894856161362, -1.70329656828, -2.78735972538, -4.44591655167, -5.28622989537, -5.71024997571,
               -1.94898449494, 2.79438767017]]),
            (0, [0.3023], [[1.03001520227]]),
            (1, [17.7, 3.854, 1.046], [[6.63856461345, 5.25433167001, 2.28748173823]]),
            (1, [0.2753], [[0.581757722201]]),
            (2, [1.185], [[3.51185437738]])],
        6: [(0, [6665.0, 1000.0, 228.0, 64.71, 21.06, 7.495, 2.797, 0.5215],
             [[1.28887278464, 2.39276233558, 4.01148824421, 5.85976508718, 6.81976661677, 5.13046804978,
               1.55679275908, 0.0235587606081],
              [-0.546552977272, -1.04144203334, -1.7047312388, -2.69921437164, -3.19078522017, -3.44781747192,
               -1.39684232934, 1.69586408122]]),
            (0, [0.1596], [[0.63795447693]]),
            (1, [9.439, 2.002, 0.5456], [[2.75016414521, 2.17593659873, 1.04017441879]]),
            (1, [0.1517], [[0.276195353793]]),
            (2, [0.55], [[0.916566737805]])],
        1: [(0, [13.01, 1.962, 0.4446], [[0.579764063557, 0.983419580181, 1.11930215022]]),
            (0, [0.122], [[0.521536727082]]),
            (1, [0.727], [[1.95840453487]])]},
    'tz': {
        8: [(0, [15330.0, 2299.0, 522.4, 147.3, 47.55, 16.76, 6.207, 0.6882],
             [[1.81067529016, 3.37486576716, 5.722654121, 8.66150357378, 10.8070275521, 9.2817953839, 3.56346172874,
               -0.0159395829751],
              [-0.686527364238, -1.28759908591, -2.19507417048, -3.43047365574, -4.58719692089, -4.89805684666,
               -2.99457591327, 1.97563930692]]),
            (0, [1.752], [[3.84738458509]]),
            (0, [0.2384], [[0.861975084244]]),
            (1, [34.46, 7.749, 2.28], [[10.0262993782, 9.72213774146, 6.55849668485]]),
            (1, [0.7156], [[1.92009319046]]),
            (1, [0.214], [[0.424621137329]]),
            (2, [2.314], [[11.3283134329]]),
            (2, [0.645], [[1.21131999657]]),
            (3, [1.428], [[4.39692267827]])],
        1: [(0, [33.87, 5.095, 1.159], [[0.904334518684, 1.63100454699, 2.40491525158]]),
            (0, [0.3258], [[1.08950275862]]),
            (0, [0.1027], [[0.458345378735]]),
            (1, [1.407], [[4.47045795164]]),
            (1, [0.388], [[0.893354952878]]),
            (2, [1.057], [[2.87515070539]])]},
}


def listed():
    return [
        # a first SCF on one molecule: host arrays through the _vhf.direct
        # drop-in, a millisecond of work in which launches count
        dict(name='jk-water-dz-host', op='jk', mol='water', n=1, basis='dz', n_dm=1, hermi=1, precision='fp64',
             side='host', delta=False),
        # an SCF iteration of a small cluster, densities kept on the GPU
        dict(name='jk-8w-dz', op='jk', mol='water', n=8, basis='dz', n_dm=1, hermi=1, precision='fp64',
             side='device', delta=False),
        # two general densities at once (UHF response, non-symmetric)
        dict(name='jk-3w-tz-2dm-general', op='jk', mol='water', n=3, basis='tz', n_dm=2, hermi=0, precision='fp64',
             side='device', delta=False),
        # a late iteration of an incremental SCF in mixed precision, odd chain
        dict(name='jk-c13-dz-mixed-delta', op='jk', mol='alkane', n=13, basis='dz', n_dm=1, hermi=1,
             precision='mixed', side='device', delta=True),
        # the triple-zeta cluster of the benchmark, a quarter of its size
        dict(name='jk-16w-tz', op='jk', mol='water', n=16, basis='tz', n_dm=1, hermi=1, precision='fp64',
             side='device', delta=False),
        # the largest: above 1500 functions the float64 defaults change
        dict(name='jk-27w-tz', op='jk', mol='water', n=27, basis='tz', n_dm=1, hermi=1, precision='fp64',
             side='device', delta=False),
        # a geometry step: E2 at new coordinates and its gradient by autograd
        dict(name='energy-7w-dz', op='energy', mol='water', n=7, basis='dz'),
        # grad.rhf.get_jk: J/K with a differentiated bra, vj and vk returned
        dict(name='gradjk-6w-dz', op='gradjk', mol='water', n=6, basis='dz', n_dm=1, side='device'),
        # the in-core SCF: fill the tensor once per geometry ...
        dict(name='fill-3w-tz', op='fill', mol='water', n=3, basis='tz'),
        # ... and contract it every iteration
        dict(name='incore-s8-192', op='incore', nao=192, sym='s8', n_dm=1, hermi=1),
        # a stored s4 matrix of an odd basis, two general densities
        dict(name='incore-s4-117-2dm', op='incore', nao=117, sym='s4', n_dm=2, hermi=0),
        # data generation: many small molecules in one build
        dict(name='batch-30-dz', op='batch', mol='water', n=30, basis='dz', precision='fp64'),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(['jk', 'jk', 'jk', 'jk', 'energy', 'gradjk', 'fill', 'incore', 'incore', 'batch'])
    basis = rng.choice(['631g', 'dz', 'dz', 'tz', 'tz'])
    if op == 'jk':
        mol = 'alkane' if basis == 'dz' and rng.random() < 0.4 else 'water'
        hermi = rng.choice([0, 1, 1, 1, 2])
        n_dm = rng.choice([1, 1, 2, 3])
        heavy = hermi != 1 or n_dm > 1
        hi = {'631g': 24, 'dz': 20, 'tz': 18}[basis] // (3 if heavy else 1)
        return dict(op=op, mol=mol, n=log_int(1, hi), basis=basis, n_dm=n_dm, hermi=hermi,
                    precision=rng.choice(['fp64', 'fp64', 'mixed']), side=rng.choice(['host', 'device']),
                    delta=rng.random() < 0.3)
    if op == 'energy':
        return dict(op=op, mol='water', n=log_int(1, {'631g': 16, 'dz': 9, 'tz': 2}[basis]), basis=basis)
    if op == 'gradjk':
        return dict(op=op, mol='water', n=log_int(1, {'631g': 16, 'dz': 9, 'tz': 2}[basis]), basis=basis,
                    n_dm=rng.choice([1, 2]), side=rng.choice(['host', 'device']))
    if op == 'fill':
        return dict(op=op, mol='water', n=log_int(1, {'631g': 12, 'dz': 7, 'tz': 3}[basis]), basis=basis)
    if op == 'incore':
        sym = rng.choice(['s8', 's8', 's4'])
        return dict(op=op, nao=log_int(13, 200 if sym == 's8' else 150), sym=sym, n_dm=rng.choice([1, 1, 2]),
                    hermi=rng.choice([0, 1, 1, 2]))
    return dict(op=op, mol='water', n=rng.randint(5, 30), basis=rng.choice(['631g', 'dz']),
                precision=rng.choice(['fp64', 'mixed']))


# ---------------------------------------------------------------------------
# molecules

def _waters(n, rng):
    """(Z, Angstrom) of n rigid waters on a cubic lattice of 3.0 Angstrom, each
    turned at random and shifted by up to 0.2 Angstrom per component."""
    h = 0.5 * math.radians(104.52)
    mono = numpy.array([[0.0, 0.0, 0.0], [0.9572 * math.sin(h), 0.0, 0.9572 * math.cos(h)],
                        [-0.9572 * math.sin(h), 0.0, 0.9572 * math.cos(h)]])
    m = 1
    while m ** 3 < n:
        m += 1
    atoms = []
    for s in range(n):
        q = rng.standard_normal(4)
        w, x, y, z = q / numpy.linalg.norm(q)
        R = numpy.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                         [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                         [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]])
        o = numpy.array([s // (m * m), s // m % m, s % m]) * 3.0 + rng.uniform(-0.2, 0.2, 3)
        atoms += [(zz, o + R @ r) for zz, r in zip((8, 1, 1), mono)]
    return atoms


def _alkane(n, rng):
    """All-trans CnH2n+2 (C-C 1.54, C-H 1.09 Angstrom, tetrahedral angles), every
    atom shifted by up to 0.02 Angstrom per component."""
    th = math.radians(109.4712)
    dx, dy = 1.54 * math.sin(th / 2), 1.54 * math.cos(th / 2)
    C = [numpy.array([i * dx, (i % 2) * dy, 0.0]) for i in range(n)]
    atoms = [(6, c) for c in C]
    for i, c in enumerate(C):
        s = 1.0 if i % 2 else -1.0
        for t in (1, -1):   # the two hydrogens of a CH2, across the backbone
            atoms.append((1, c + 1.09 * numpy.array([0.0, s * math.cos(th / 2), t * math.sin(th / 2)])))
        for end, sign in ((0, -1.0), (n - 1, 1.0)):
            if i == end:    # the end hydrogen continues the zig-zag
                atoms.append((1, c + 1.09 * numpy.array([sign * math.sin(th / 2), -s * math.cos(th / 2), 0.0])))
    return [(z, r + rng.uniform(-0.02, 0.02, 3)) for z, r in atoms]


def _molecule(case, rng, n=None):
    """PySCF's atm, bas, env of the case's molecule, and its nao."""
    n = case['n'] if n is None else n
    atoms = _alkane(n, rng) if case['mol'] == 'alkane' else _waters(n, rng)
    env = [0.0] * 20
    atm, bas, where = [], [], {}
    for z, r in atoms:
        atm.append([z, len(env), 1, len(env) + 3, 0, 0])
        env += [float(x) / BOHR for x in r] + [0.0]
    nao = 0
    for ia, (z, _) in enumerate(atoms):
        for k, (l, e, c) in enumerate(BASIS[case['basis']][z]):
            if (z, k) not in where:
                where[z, k] = (len(env), len(env) + len(e))
                env += e + [x for col in c for x in col]
            bas.append([ia, l, len(e), len(c), 0, where[z, k][0], where[z, k][1], 0])
            nao += (2 * l + 1) * len(c)
    return numpy.array(atm, dtype=numpy.int32), numpy.array(bas, dtype=numpy.int32), numpy.array(env), nao


def _densities(nao, n_dm, hermi, delta, rng):
    """Occupied-orbital densities C C^T (hermi 1), C C'^T (0) or their
    antisymmetric part (2); delta: the small change of a late iteration."""
    out = []
    for _ in range(n_dm):
        c = rng.standard_normal((nao, max(1, nao // 5))) / math.sqrt(nao)
        d = c @ c.T
        if hermi != 1:
            d = c @ (c + 0.3 * rng.standard_normal(c.shape) / math.sqrt(nao)).T
        if hermi == 2:
            d = d - d.T
        out.append(1e-4 * d if delta else d)
    return numpy.array(out)


class _Mol:
    def __init__(self, atm, bas, env):
        self._atm, self._bas, self._env, self.cart = atm, bas, env, False


def _inputs(case, seed):
    """Molecule and densities of the ops that work on one molecule."""
    rng = numpy.random.default_rng(seed)
    atm, bas, env, nao = _molecule(case, rng)
    dms = _densities(nao, case.get('n_dm', 1), case.get('hermi', 1), case.get('delta', False), rng)
    return atm, bas, env, nao, dms


def _incore_inputs(case, seed):
    """A stored tensor with the spread of a molecule's integrals (products of
    pair bounds over six decades) and densities, on the GPU."""
    g = torch.Generator(device='cuda').manual_seed(seed)
    nao = case['nao']
    npair = nao * (nao + 1) // 2
    q = torch.exp(torch.rand(npair, generator=g, device='cuda', dtype=torch.float64) * -7.0)
    if case['sym'] == 's4':
        m = torch.rand((npair, npair), generator=g, device='cuda', dtype=torch.float64).mul_(2.0).sub_(1.0)
        m += m.T.clone()
        eri = m.mul_(0.5 * q[:, None]).mul_(q[None, :])
    else:
        eri = torch.rand(npair * (npair + 1) // 2, generator=g, device='cuda', dtype=torch.float64).mul_(2.0).sub_(1.0)
        for p in range(npair):
            eri[p * (p + 1) // 2:(p + 1) * (p + 2) // 2].mul_(q[p] * q[:p + 1])
    dms = torch.from_numpy(_densities(nao, case['n_dm'], case['hermi'], False, numpy.random.default_rng(seed))).cuda()
    return eri, dms


def prepare(case, seed):
    op = case['op']
    s = dict(case)
    if op == 'incore':
        s['eri'], s['dms'] = _incore_inputs(case, seed)
        return s
    if op == 'batch':
        rng = numpy.random.default_rng(seed)
        sizes = [1 + (3 * k) % 16 for k in range(case['n'])]
        mols = [_molecule(case, rng, n) for n in sizes]
        s['batch'] = lib.Batch([lib.Plan(a, b, e) for a, b, e, _ in mols])
        s['dms'] = [torch.from_numpy(_densities(nao, 1, 1, False, rng)[0]).cuda() for _, _, _, nao in mols]
        return s
    atm, bas, env, nao, dms = _inputs(case, seed)
    if op == 'jk':
        if case['side'] == 'host' and case['precision'] == 'fp64':
            s['mol'], s['opt'] = (atm, bas, env), _vhf.VHFOpt(_Mol(atm, bas, env))
        else:
            s['plan'] = lib.Plan(atm, bas, env)
        s['dms'] = dms if case['side'] == 'host' else torch.from_numpy(dms).cuda()
    elif op == 'energy':
        coords = numpy.array([env[a[1]:a[1] + 3] for a in atm])
        s['coords'], s['dms'] = torch.from_numpy(coords).requires_grad_(True), torch.from_numpy(dms[0]).cuda()
        s['dms'].requires_grad_(True)
        s['mol'] = (atm, bas, env)
    else:
        s['plan'] = lib.Plan(atm, bas, env)
        if op == 'gradjk':
            s['dms'] = dms if case['side'] == 'host' else torch.from_numpy(dms).cuda()
    return s


def run(s):
    # (the J of an antisymmetric density is zero: hermi 2 builds K alone)
    op = s['op']
    if op == 'jk':
        if 'opt' in s:
            return list(_vhf.direct(s['dms'], *s['mol'], vhfopt=s['opt'], hermi=s['hermi'], with_j=s['hermi'] != 2))
        build = s['plan'].get_jk if s['side'] == 'host' else s['plan'].get_jk_device
        return list(build(s['dms'], hermi=s['hermi'], with_j=s['hermi'] != 2,
                          precision=lib.PREC_MIXED if s['precision'] == 'mixed' else lib.PREC_FP64))
    if op == 'energy':
        e = grad.two_electron_energy(s['coords'], s['dms'], *s['mol'])
        return [e.detach(), *torch.autograd.grad(e, [s['coords'], s['dms']])]
    if op == 'gradjk':
        return list((s['plan'].grad_jk if s['side'] == 'host' else s['plan'].grad_jk_device)(s['dms']))
    if op == 'fill':
        return s['plan'].int2e_s8()
    if op == 'incore':
        return list(incore.incore(s['eri'], s['dms'], s['hermi'], with_j=s['hermi'] != 2))
    vj, vk = s['batch'].get_jk_device(s['dms'],
                                      precision=lib.PREC_MIXED if s['precision'] == 'mixed' else lib.PREC_FP64)
    return vj + vk


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _quartets(case, n=None):
    """[(class, quartets, primitive quartets)] that survive an estimate of the
    1e-13 Schwarz screen (bounds of the most diffuse s pair) at seed 0."""
    atm, bas, env, _ = _molecule(case, numpy.random.default_rng(0), n)
    seg = [(int(b[1]), env[b[5]:b[5] + b[2]], env[atm[b[0]][1]:atm[b[0]][1] + 3]) for b in bas for _ in range(b[3])]
    pairs = {}
    for i, (li, ei, ri) in enumerate(seg):
        for lj, ej, rj in seg[:i + 1]:
            rr = float(((ri - rj) ** 2).sum())
            a, b = ei.min(), ej.min()
            o = (2.0 * math.sqrt(a * b) / (a + b)) ** 1.5 * math.exp(-min(300.0, a * b / (a + b) * rr))
            bound = o * math.sqrt(2.0 * math.sqrt((a + b) / (2.0 * math.pi)))
            prim = int(((ei[:, None] * ej / (ei[:, None] + ej)) * rr < 60.0).sum())
            pairs.setdefault((max(li, lj), min(li, lj)), []).append((bound, prim))
    out = []
    keys = sorted(pairs)
    tab = {k: tuple(numpy.array(v) for v in zip(*sorted(pairs[k], reverse=True))) for k in keys}
    for x, X in enumerate(keys):
        for Y in keys[:x + 1]:
            (qx, px), (qy, py) = tab[X], tab[Y]
            cum = numpy.concatenate([[0.0], numpy.cumsum(py)])
            cnt = numpy.searchsorted(-qy, -1e-13 / numpy.maximum(qx, 1e-300))
            half = 0.5 if X == Y else 1.0
            out.append((X + Y, half * cnt.sum(), half * (px * cum[cnt]).sum()))
    return out


def _nao(case, n=None):
    return _molecule(case, numpy.random.default_rng(0), n)[3]


def _jk_work(case, n=None):
    n_dm = case.get('n_dm', 1)
    nk = 1 if case.get('hermi', 1) == 1 else 2
    nao = _nao(case, n)
    f = sum(np_ * flops.prim_quartet_flops(*c) + nq * n_dm * (4 + 8 * nk) * _ng(c) for c, nq, np_ in _quartets(case, n))
    return 24.0 * n_dm * nao * nao, f


def _ng(c):
    return math.prod(flops.ncart(l) for l in c)


def _grad_work(case):
    """One bra centre raised by a derivative on either side of a quartet."""
    f = 0.0
    for c, nq, np_ in _quartets(case):
        f += np_ * 2.0 * flops.prim_quartet_flops(c[0] + 1, *c[1:]) + nq * 6 * 12.0 * _ng(c)
    return f


def work(case):
    op = case['op']
    if op == 'jk':
        b, f = _jk_work(case)
    elif op == 'batch':
        both = [_jk_work(case, 1 + (3 * k) % 16) for k in range(case['n'])]
        b, f = sum(x[0] for x in both), sum(x[1] for x in both)
    elif op == 'energy':
        b, f = _jk_work(case)
        f += _grad_work(case)
    elif op == 'gradjk':
        nao = _nao(case)
        b, f = 8.0 * case['n_dm'] * nao * nao * 7, _grad_work(case)
    elif op == 'fill':
        npair = _nao(case) * (_nao(case) + 1) // 2
        b = 4.0 * npair * (npair + 1)
        f = sum(np_ * flops.prim_quartet_flops(*c) for c, _, np_ in _quartets(case))
    else:
        nao, n_dm, nk = case['nao'], case['n_dm'], 2 if case['hermi'] == 0 else 1
        npair = nao * (nao + 1) // 2
        entries = npair * (npair + 1) // 2 if case['sym'] == 's8' else npair * npair
        b = 8.0 * entries + 24.0 * n_dm * nao * nao
        f = entries * n_dm * (4.0 + 8.0 * nk)
    return {'bytes': b, 'flops': f}


# ---------------------------------------------------------------------------
# independent results: McMurchie-Davidson integrals of small molecules, and
# the plain contraction of a stored tensor

SPH = {0: numpy.array([[0.282094791773878143]]),
       1: 0.488602511902919921 * numpy.eye(3),
       2: numpy.array([[0, 1.09254843059207907, 0, 0, 0, 0], [0, 0, 0, 0, 1.09254843059207907, 0],
                       [-0.31539156525252, 0, 0, -0.31539156525252, 0, 0.63078313050504],
                       [0, 0, 1.09254843059207907, 0, 0, 0],
                       [0.54627421529603954, 0, 0, -0.54627421529603954, 0, 0]])}


def _cart(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _e_coef(la, lb, a, b, d):
    """Hermite expansion coefficients E[i][j][t] of one direction, d = A - B."""
    p = a + b
    E = numpy.zeros((la + 1, lb + 1, la + lb + 2))
    E[0, 0, 0] = math.exp(-a * b / p * d * d)
    for i in range(la + 1):
        for j in range(lb + 1):
            if i + j == 0:
                continue
            src, shift = (E[i - 1, j], -b / p * d) if i else (E[i, j - 1], a / p * d)
            for t in range(i + j + 1):
                E[i, j, t] = shift * src[t] + (t + 1) * src[t + 1] + (src[t - 1] / (2 * p) if t else 0.0)
    return E


def _eri(atm, bas, env, nao):
    """The whole (nao^2, nao^2) integral matrix, or None where it is not small."""
    shells, off = [], 0
    for b in bas:
        l, np_, nc = int(b[1]), int(b[2]), int(b[3])
        e, c = env[b[5]:b[5] + np_], env[b[6]:b[6] + np_ * nc].reshape(nc, np_)
        shells += [(l, e[k], env[atm[b[0]][1]:atm[b[0]][1] + 3], c[:, k], off) for k in range(np_)]
        off += (2 * l + 1) * nc
    lmax = max(s[0] for s in shells)
    herm = [(x, y, z) for x in range(2 * lmax + 1) for y in range(2 * lmax + 1 - x) for z in range(2 * lmax + 1 - x - y)]
    nh, npr = len(herm), len(shells) * (len(shells) + 1) // 2
    if lmax > 2 or nh * npr > 14000:
        return None
    dev = 'cuda' if torch.cuda.is_available() else 'cpu'
    B = numpy.zeros((nao * nao, npr, nh))
    P, pe = numpy.zeros((npr, 3)), numpy.zeros(npr)
    k = 0
    for i, (li, a, ri, ci, oi) in enumerate(shells):
        for j, (lj, b, rj, cj, oj) in enumerate(shells[:i + 1]):
            pe[k], P[k] = a + b, (a * ri + b * rj) / (a + b)
            E = [_e_coef(li, lj, a, b, ri[x] - rj[x]) for x in range(3)]
            block = numpy.array([[[E[0][u[0], v[0], h[0]] * E[1][u[1], v[1], h[1]] * E[2][u[2], v[2], h[2]]
                                   if all(h[x] <= u[x] + v[x] for x in range(3)) else 0.0 for h in herm]
                                  for v in _cart(lj)] for u in _cart(li)])
            block = numpy.einsum('mu,uvh,nv->mnh', SPH[li], block, SPH[lj])
            for x, cx in enumerate(ci):
                for y, cy in enumerate(cj):
                    for m in range(2 * li + 1):
                        for q in range(2 * lj + 1):
                            mu, nu = oi + x * (2 * li + 1) + m, oj + y * (2 * lj + 1) + q
                            B[mu * nao + nu, k] += cx * cy * block[m, q]
                            if i != j:
                                B[nu * nao + mu, k] += cx * cy * block[m, q]
            k += 1
    L = 4 * lmax
    P, pe, B = (torch.from_numpy(v).to(dev) for v in (P, pe, B))
    sign = torch.tensor([(-1.0) ** sum(h) for h in herm], dtype=torch.float64, device=dev)
    at = {}
    for h in herm:
        for g in herm:
            at.setdefault(tuple(x + y for x, y in zip(h, g)), len(at))
    sel = torch.tensor([[at[tuple(x + y for x, y in zip(h, g))] for g in herm] for h in herm], device=dev).reshape(-1)
    eri = torch.zeros((nao * nao, nao * nao), dtype=torch.float64, device=dev)
    step = max(1, int(2e8) // (npr * nh * nh * 8))
    for k0 in range(0, npr, step):
        p = pe[k0:k0 + step, None]
        X = P[k0:k0 + step, None, :] - P[None]
        al = p * pe / (p + pe)
        T = al * (X * X).sum(-1)
        # Boys function: series of the highest order (positive terms), its
        # limit beyond T = 100, downward recurrence
        Ts, term = T.clamp(max=100.0), torch.full_like(T, 1.0 / (2 * L + 1))
        F = term.clone()
        for m in range(1, 330):
            term = term * (2 * Ts / (2 * L + 2 * m + 1))
            F += term
        F = F * torch.exp(-Ts)
        F = torch.where(T > 100.0, math.gamma(L + 0.5) / 2 / T.clamp(min=1.0) ** (L + 0.5), F)
        boys = [None] * L + [F]
        for m in range(L - 1, -1, -1):
            boys[m] = (2 * T * boys[m + 1] + torch.exp(-T)) / (2 * m + 1)
        R = {(0, 0, 0): [(-2 * al) ** m * boys[m] for m in range(L + 1)]}
        for t in sorted(at, key=sum):
            if t in R:
                continue
            x = max(range(3), key=lambda y: t[y])
            one = tuple(v - (y == x) for y, v in enumerate(t))
            two = tuple(v - 2 * (y == x) for y, v in enumerate(t))
            R[t] = [X[..., x] * R[one][m + 1] + ((t[x] - 1) * R[two][m + 1] if t[x] > 1 else 0.0)
                    for m in range(L + 1 - sum(t))]
        pref = 2 * math.pi ** 2.5 / (p * pe * torch.sqrt(p + pe))
        V = torch.stack([R[t][0] * pref for t in at], -1)[..., sel].reshape(p.shape[0], npr, nh, nh) * sign
        V = V.permute(0, 2, 1, 3).reshape(p.shape[0] * nh, npr * nh)
        eri += B[:, k0:k0 + step].reshape(nao * nao, -1) @ (V @ B.reshape(nao * nao, -1).T)
    return eri


def _full_rows(case, eri, i):
    """(ij|kl) of one i, (nao, nao, nao), from the stored tensor."""
    nao = case['nao']
    npair = nao * (nao + 1) // 2
    a = torch.arange(nao, device=eri.device)
    hi, lo = torch.maximum(a[:, None], a), torch.minimum(a[:, None], a)
    tri = hi * (hi + 1) // 2 + lo
    p = tri[i]
    if case['sym'] == 's4':
        return eri[p][:, tri]
    q = torch.arange(npair, device=eri.device)
    big, small = torch.maximum(p[:, None], q), torch.minimum(p[:, None], q)
    return eri[big * (big + 1) // 2 + small][:, tri]


def exact(case, seed):
    op = case['op']
    if op == 'incore':
        eri, dms = _incore_inputs(case, seed)
        nao = case['nao']
        vj, vk = torch.zeros_like(dms), torch.zeros_like(dms)
        for i in range(nao):
            v = _full_rows(case, eri, i)
            for s in range(case['n_dm']):
                vj[s, i] = (v.reshape(nao, -1) @ dms[s].T.reshape(-1))
                vk[s, i] = torch.einsum('jkl,jk->l', v, dms[s])
        return [vj, vk] if case['hermi'] != 2 else [None, vk]
    if op not in ('jk', 'fill'):
        return None
    atm, bas, env, nao, dms = _inputs(case, seed)
    if nao > 40:
        return None
    eri = _eri(atm, bas, env, nao)
    if eri is None:
        return None
    if op == 'fill':
        a, b = torch.tril_indices(nao, nao, device=eri.device)
        m = eri[a * nao + b][:, a * nao + b]
        x, y = torch.tril_indices(m.shape[0], m.shape[0], device=eri.device)
        return m[x, y]
    d = torch.from_numpy(dms).to(eri.device)
    e4 = eri.reshape(nao, nao, nao, nao)
    out = [torch.einsum('ijkl,sji->skl', e4, d), torch.einsum('ijkl,sjk->sil', e4, d)]
    out = [x.cpu().numpy() if case['side'] == 'host' else x for x in out]
    return out if case['hermi'] != 2 else [None, out[1]]
