"""Timed cases of the framework: the work that an SCF on the wB97M-V /
COSX(pjs) path has it do, through its public entry points.

Kinds (``case['kind']``):

* ``k``      exchange build of one SCF cycle, both omegas
             (CosxEngine.get_k_multi): every cycle of the FP32 stages;
* ``k1``     the same for one omega (CosxEngine.get_k): what the PySCF hook
             asks for when it wants one operator only;
* ``batch``  exchange builds of several molecules of uneven size in one call
             (CosxBatch.run): lockstep SCFs;
* ``k64``    the plain FP64 exchange build (CosxEngine.get_k_fp64): the FP64
             tail of a staged SCF and the plain FP64 SCF;
* ``grad``   exchange nuclear gradient (CosxEngine.k_grad): one per geometry
             of an optimisation or a trajectory;
* ``xc``     semilocal exchange-correlation of one cycle (gpu_nr_rks), the
             functional on the host as in PySCF;
* ``vv10``   non-local correlation of one cycle (gpu_nr_nlc_vxc);
* ``fock``   a whole Fock build of the device SCF (DeviceRKS.fock), in the
             FP32 form of the stages or the plain FP64 form.

Molecules are the seeded water clusters (def2-SVP structure) and the
all-trans n-alkanes (def2-TZVP structure, f shells) of the repository's own
tests and benchmark, grids its own Becke grids.  The density is
2 C C^T with C seeded, localised orbitals (each centred on an atom and
decaying with the distance from it, as occupied orbitals of a molecule with
a gap do).
"""
import functools
import math
import types

import numpy as np
import torch

from pyscf_wb97mv_fast_gb300.basis import ANGSTROM, Molecule
from pyscf_wb97mv_fast_gb300.cosx import (CosxBatch, CosxEngine,
                                          model_flops_per_point)
from pyscf_wb97mv_fast_gb300.gpu.vv10 import Vv10Context, gpu_nr_nlc_vxc
from pyscf_wb97mv_fast_gb300.gpu.xc import XcContext, gpu_nr_rks
from pyscf_wb97mv_fast_gb300.grids import GRID_LEVELS, build_grids
from pyscf_wb97mv_fast_gb300.scf import DeviceGrid, DeviceRKS
from pyscf_wb97mv_fast_gb300.systems import alkane, water_cluster

OMEGAS = (0.0, 0.3)
NLC_PARS = (6.0, 0.01)


# -- the cases -------------------------------------------------------------------

def listed():
    return [
        # latency end: a water dimer's exchange build on the coarse grid
        dict(name='k_water2', kind='k', mol='water', n=2, level=0, geom=1),
        # the benchmark's cluster and grid: 27 waters, 648 AOs, 3.8e5 points
        dict(name='k_water27', kind='k', mol='water', n=27, level=2, geom=27),
        # long-range exchange alone, f shells, ragged class sizes
        dict(name='k1_alkane8', kind='k1', mol='alkane', n=8, level=1, omega=0.3),
        # lockstep SCFs of uneven clusters on coarse grids
        dict(name='batch_water', kind='batch', sizes='4,5,7,9,12,17', level=0, geom=5),
        # FP64 tail of the small-cluster SCF
        dict(name='k64_water8', kind='k64', mol='water', n=8, level=1, geom=8),
        # exchange gradients: light shells, and f shells with odd sizes
        dict(name='grad_water8', kind='grad', mol='water', n=8, level=0, geom=8,
             omega=0.0),
        dict(name='grad_alkane4', kind='grad', mol='alkane', n=4, level=0, omega=0.3),
        # semilocal meta-GGA of a middle-sized cluster
        dict(name='xc_water16', kind='xc', mol='water', n=16, level=2, geom=16,
             xctype='MGGA'),
        # VV10 on the small cluster's NLC grid, and on a fine alkane grid
        dict(name='vv10_water8', kind='vv10', mol='water', n=8, level=1, geom=8,
             tile_tol=0.0),
        dict(name='vv10_alkane10', kind='vv10', mol='alkane', n=10, level=2, tile_tol=0.0),
        # whole Fock builds: the FP32 stages' and the plain FP64 form's
        dict(name='fock_water8', kind='fock', mol='water', n=8, geom=8, xc=2, sgx=1,
             nlc=1, fp64=False),
        dict(name='fock64_water4', kind='fock', mol='water', n=4, geom=4, xc=1, sgx=0,
             nlc=0, fp64=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(('k', 'k', 'k1', 'batch', 'k64', 'grad', 'xc', 'vv10', 'fock'))
    if kind == 'batch':
        k = rng.randint(2, 6)
        return dict(kind=kind, sizes=','.join(str(_log_int(rng, 2, 17)) for _ in range(k)),
                    level=0, geom=rng.randrange(1000))
    case = dict(kind=kind)
    # (waters, water levels), (carbons, alkane levels)
    waters, wl, carbons, al = {
        'k': ((2, 27), (0, 1, 2), (2, 10), (0, 1)),
        'k1': ((2, 27), (0, 1, 2), (2, 10), (0, 1)),
        'k64': ((2, 8), (0, 1), (2, 4), (0,)),
        'grad': ((2, 8), (0,), (2, 4), (0,)),
        'xc': ((2, 16), (1, 2), (2, 8), (1,)),
        'vv10': ((2, 16), (0, 1, 2), (2, 10), (0, 1, 2)),
        'fock': ((2, 8), (0, 1), (2, 4), (0,)),
    }[kind]
    if rng.random() < 0.6:
        case.update(mol='water', n=_log_int(rng, *waters), level=rng.choice(wl),
                    geom=rng.randrange(1000))
    else:
        case.update(mol='alkane', n=_log_int(rng, *carbons), level=rng.choice(al))
    if kind == 'k1' or kind == 'grad':
        case['omega'] = rng.choice(OMEGAS)
    elif kind == 'xc':
        case['xctype'] = rng.choice(('GGA', 'MGGA', 'MGGA'))
    elif kind == 'vv10':
        case['tile_tol'] = rng.choice((0.0, 0.0, 1e-12, 1e-10))
    elif kind == 'fock':
        lv = case.pop('level')
        case.update(xc=lv + 1, sgx=lv, nlc=lv, fp64=rng.random() < 0.4 and case['n'] <= 4)
    return case


# -- what a program has in hand ----------------------------------------------------

@functools.lru_cache(maxsize=8)
def _water(n, geom):
    return Molecule.build(water_cluster(n, box=max(5.0, 3.4 * n ** (1.0 / 3.0)), seed=geom),
                          'synthetic-svp')


@functools.lru_cache(maxsize=8)
def _alkane(n):
    return Molecule.build(alkane(n), 'synthetic-tzvp')


def _molecule(case):
    return _water(case['n'], case['geom']) if case['mol'] == 'water' else _alkane(case['n'])


@functools.lru_cache(maxsize=8)
def _water_grid(n, geom, level):
    return build_grids(_water(n, geom), level=level)


@functools.lru_cache(maxsize=8)
def _alkane_grid(n, level):
    return build_grids(_alkane(n), level=level)


def _grid(case, level):
    if case['mol'] == 'water':
        return _water_grid(case['n'], case['geom'], level)
    return _alkane_grid(case['n'], level)


def _batch_sizes(case):
    return [int(n) for n in case['sizes'].split(',')]


def _density(mol, seed):
    """2 C C^T (host FP64) with nelectron / 2 seeded localised orbitals."""
    rng = np.random.default_rng(seed)
    nocc = max(1, mol.nelectron // 2)
    xyz = mol.atom_coords()
    heavy = np.argsort(-mol.atom_charges(), kind='stable')
    centre = xyz[heavy[np.arange(nocc) % len(heavy)]]
    owner = np.concatenate([[sh.atom] * sh.nao for sh in mol.shells])
    far = np.linalg.norm(xyz[owner][:, None] - centre[None], axis=2)
    c = rng.normal(size=(mol.nao, nocc)) * np.exp(-far / (1.2 * ANGSTROM))
    c /= np.linalg.norm(c, axis=0)
    return 2.0 * c @ c.T


class _Numint:
    """The pieces of PySCF's NumInt that the flows read."""

    def __init__(self, xctype='MGGA'):
        self.xctype = xctype

    def _xc_type(self, xc_code):
        return self.xctype

    def nlc_coeff(self, xc_code):
        return ((NLC_PARS, 1.0),)


class _Functional:
    """A smooth model functional in the libxc convention:
    e = -0.7386 rho^(4/3) - 0.01 sigma / (0.1 + rho) [+ 0.02 tau rho / (1 + rho)]
    per volume."""

    def __init__(self, xctype):
        self.mgga = xctype == 'MGGA'

    def eval(self, rho):
        r = np.maximum(rho[0], 1e-14)
        sigma = (rho[1:4] ** 2).sum(axis=0)
        third = np.cbrt(r)
        q = 1.0 / (0.1 + r)
        e = -0.7386 * r * third - 0.01 * sigma * q
        vrho = -0.7386 * 4.0 / 3.0 * third + 0.01 * sigma * q * q
        vsigma = -0.01 * q
        vtau = None
        if self.mgga:
            s = 1.0 / (1.0 + r)
            e = e + 0.02 * rho[4] * r * s
            vrho = vrho + 0.02 * rho[4] * s * s
            vtau = 0.02 * r * s
        return e / r, vrho, vsigma, vtau


def prepare(case, seed):
    kind = case['kind']
    dev = torch.device('cuda')
    s = types.SimpleNamespace(kind=kind, case=case)
    if kind == 'batch':
        engines, grids, s.qds = [], [], []
        for i, n in enumerate(_batch_sizes(case)):
            mol = _water(n, case['geom'] + i)
            g = _water_grid(n, case['geom'] + i, case['level'])
            eng = CosxEngine(mol)
            engines.append(eng)
            grids.append((eng.relative(g.coords), torch.as_tensor(g.weights, device=dev)))
            s.qds.append(torch.as_tensor(_density(mol, seed + 1000 * i), device=dev))
        s.batch = CosxBatch(engines, grids, OMEGAS)
        return s
    mol = _molecule(case)
    dm = _density(mol, seed)
    if kind in ('xc', 'vv10'):
        s.mol, s.dm = mol, dm
        s.grids = _grid(case, case['level'])
        if kind == 'xc':
            s.ni = _Numint(case['xctype'])
            s.ctx = XcContext(mol, functional_factory=lambda xc, ni: _Functional(ni.xctype))
        else:
            s.ni = _Numint()
            s.ctx = Vv10Context(mol, tile_tol=case['tile_tol'])
        s.ctx.build()
        return s
    s.dm = torch.as_tensor(dm, device=dev)
    if kind == 'fock':
        s.rks = DeviceRKS(mol)
        s.grids = {k: DeviceGrid(s.rks.eng, _grid(case, case[k]), deriv=1 if k == 'nlc' else 0)
                   for k in ('xc', 'sgx', 'nlc')}
        return s
    s.eng = CosxEngine(mol)
    g = _grid(case, case['level'])
    s.coords = s.eng.relative(g.coords)
    s.weights = torch.as_tensor(g.weights, device=dev)
    return s


def run(s):
    c = s.case
    if s.kind == 'k':
        return s.eng.get_k_multi(s.coords, s.weights, s.dm, OMEGAS, stats=False)
    if s.kind == 'k1':
        return s.eng.get_k(s.coords, s.weights, s.dm, c['omega'], stats=False)
    if s.kind == 'batch':
        return s.batch.run(s.qds)
    if s.kind == 'k64':
        return s.eng.get_k_fp64(s.coords, s.weights, s.dm, OMEGAS, stats=False)
    if s.kind == 'grad':
        return s.eng.k_grad(s.coords, s.weights, s.dm, c['omega'], tile_tol=1e-11)
    if s.kind == 'xc':
        return gpu_nr_rks(s.ctx, s.ni, s.mol, s.grids, 'model', s.dm)
    if s.kind == 'vv10':
        return gpu_nr_nlc_vxc(s.ctx, s.ni, s.mol, s.grids, 'model', s.dm)
    E, F, parts, _ = s.rks.fock(s.dm, s.grids, c['fp64'])
    return dict(parts, E=E, F=F)


# -- what a pass cannot do without ---------------------------------------------------

def _points(mol, level):
    """Grid points before the pruning of negligible weights."""
    nh, nx, nt = GRID_LEVELS[level]
    return sum((nh if s == 'H' else nx) * 2 * nt * nt for s in mol.symbols)


def _k_work(mol, level, omegas, derivative=1.0):
    n, nao = _points(mol, level), mol.nao
    # integrals and their contraction by the model count of every shell pair
    # (the screen drops part of it), F = X D and K = X^T (w G)
    flops = model_flops_per_point(mol)[0] * n * omegas * derivative
    flops += 2.0 * n * nao * nao * (1 + omegas)
    return 32.0 * n + 8.0 * nao * nao * (1 + omegas), flops


def _xc_work(mol, level, planes):
    n, nao = _points(mol, level), mol.nao
    return 32.0 * n + 16.0 * nao * nao, 4.0 * planes * n * nao * nao


def _vv10_work(mol, level):
    n, nao = _points(mol, level), mol.nao
    return 32.0 * n + 16.0 * nao * nao, 27.0 * n * n + 4.0 * n * nao * nao


def work(case):
    kind = case['kind']
    if kind == 'batch':
        parts = [_k_work(_water(n, case['geom'] + i), case['level'], 2)
                 for i, n in enumerate(_batch_sizes(case))]
        return {'bytes': sum(p[0] for p in parts), 'flops': sum(p[1] for p in parts)}
    mol = _molecule(case)
    if kind == 'xc':
        b, f = _xc_work(mol, case['level'], 4 if case['xctype'] == 'MGGA' else 1)
    elif kind == 'vv10':
        b, f = _vv10_work(mol, case['level'])
    elif kind == 'fock':
        parts = [_k_work(mol, case['sgx'], 2), _xc_work(mol, case['xc'], 1),
                 _vv10_work(mol, case['nlc'])]
        b, f = (sum(p[i] for p in parts) for i in (0, 1))
    else:
        b, f = _k_work(mol, case['level'], 1 if kind in ('k1', 'grad') else 2,
                       3.0 if kind == 'grad' else 1.0)
    return {'bytes': b, 'flops': f}


# -- the same quantities in plain 64-bit torch ---------------------------------------
#
# Real solid harmonics (unit sphere) per l in the order of the AO columns:
# {(i, j, k): coefficient of x^i y^j z^k}.
_D = 0.31539156525252005
_F0, _F1, _F3 = 0.3731763325901154, 0.4570457994644658, 0.5900435899266435
_SOLID = (
    ({(0, 0, 0): 0.28209479177387814},),
    tuple({e: 0.4886025119029199} for e in ((1, 0, 0), (0, 1, 0), (0, 0, 1))),
    ({(1, 1, 0): 1.0925484305920792}, {(0, 1, 1): 1.0925484305920792},
     {(0, 0, 2): 2 * _D, (2, 0, 0): -_D, (0, 2, 0): -_D}, {(1, 0, 1): 1.0925484305920792},
     {(2, 0, 0): 0.5462742152960396, (0, 2, 0): -0.5462742152960396}),
    ({(2, 1, 0): 3 * _F3, (0, 3, 0): -_F3}, {(1, 1, 1): 2.890611442640554},
     {(0, 1, 2): 4 * _F1, (2, 1, 0): -_F1, (0, 3, 0): -_F1},
     {(0, 0, 3): 2 * _F0, (2, 0, 1): -3 * _F0, (0, 2, 1): -3 * _F0},
     {(1, 0, 2): 4 * _F1, (3, 0, 0): -_F1, (1, 2, 0): -_F1},
     {(2, 0, 1): 1.445305721320277, (0, 2, 1): -1.445305721320277},
     {(3, 0, 0): _F3, (1, 2, 0): -3 * _F3}),
)
_CART = [[(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]
         for l in range(4)]


def _ao(mol, xyz, atoms, deriv=False):
    """AO values (nao, P) at xyz (P, 3), atoms (natm, 3), and with deriv their
    x, y, z derivatives: (4, nao, P)."""
    rows = []
    for sh in mol.shells:
        d = xyz - atoms[sh.atom]
        r2 = (d * d).sum(dim=1)
        rad, drad = 0.0, 0.0
        for a, c in zip(sh.exps, sh.coeffs[:, 0]):
            e = float(c) * torch.exp(-float(a) * r2)
            rad, drad = rad + e, drad - 2.0 * float(a) * e
        for poly in _SOLID[sh.l]:
            mono = lambda e: d[:, 0] ** e[0] * d[:, 1] ** e[1] * d[:, 2] ** e[2]  # noqa: E731
            val = sum(c * mono(e) for e, c in poly.items())
            out = [rad * val]
            for x in range(3) if deriv else ():
                g = sum(c * e[x] * mono([v - (i == x) for i, v in enumerate(e)])
                        for e, c in poly.items() if e[x])
                out.append(rad * g + drad * val * d[:, x])
            rows.append(torch.stack(out) if deriv else out[0])
    return torch.stack(rows, dim=1 if deriv else 0)


@functools.lru_cache(maxsize=2)
def _boys_table(device):
    """F_n(k / 8), n < 24, k / 8 < 36: the ascending series (Helgaker,
    Jorgensen, Olsen, Molecular Electronic-Structure Theory, 9.8.11)."""
    t = np.arange(8 * 36 + 1)[:, None] / 8.0
    n = np.arange(24)[None, :]
    term = np.exp(-t) / (2 * n + 1)
    total = term.copy()
    for i in range(1, 260):
        term = term * 2 * t / (2 * n + 2 * i + 1)
        total += term
    return torch.as_tensor(total, device=device)


def _boys(T, L):
    """F_0 .. F_L: Taylor series about the nearest node and downward
    recursion below 35, the asymptotic form and upward recursion above."""
    tab = _boys_table(str(T.device))
    Tn = T.clamp(max=35.0)
    k = torch.round(Tn.detach() * 8.0)
    x = k / 8.0 - Tn
    k = k.long()
    near = tab[:, L + 11][k] * (x / 11.0)
    for j in range(10, 0, -1):
        near = (tab[:, L + j][k] + near) * (x / j)
    near = [tab[:, L][k] + near]
    e = torch.exp(-Tn)
    for n in range(L - 1, -1, -1):
        near.insert(0, (2.0 * Tn * near[0] + e) / (2 * n + 1))
    Tf = T.clamp(min=35.0)
    ef = torch.exp(-Tf)
    far = [0.5 * math.sqrt(math.pi) * torch.rsqrt(Tf)]
    for n in range(L):
        far.append(((2 * n + 1) * far[-1] - ef) / (2.0 * Tf))
    return [torch.where(T < 35.0, a, b) for a, b in zip(near, far)]


def _hermite(la, lb, p, xpa, xpb):
    """E^{ij}_t of one axis, {(i, j, t): tensor}."""
    E = {(0, 0, 0): torch.ones_like(p)}
    get = lambda i, j, t: E.get((i, j, t), 0.0)  # noqa: E731
    for i in range(la + 1):
        for j in range(lb + 1):
            if i + j == 0:
                continue
            pi, pj, x = (i - 1, j, xpa) if i else (i, j - 1, xpb)
            for t in range(i + j + 1):
                E[i, j, t] = (get(pi, pj, t - 1) / (2.0 * p) + x * get(pi, pj, t)
                              + (t + 1) * get(pi, pj, t + 1))
    return E


def _hermite_coulomb(L, F, alpha, X, Y, Z):
    """R_tuv, t + u + v <= L (McMurchie and Davidson, 1978)."""
    cur = {}
    for n in range(L, -1, -1):
        new = {(0, 0, 0): (-2.0 * alpha) ** n * F[n]}
        for m in range(1, L - n + 1):
            for t in range(m, -1, -1):
                for u in range(m - t, -1, -1):
                    v = m - t - u
                    e = [t, u, v]
                    ax = 0 if t else 1 if u else 2
                    c = (X, Y, Z)[ax]
                    e[ax] -= 1
                    val = c * cur[tuple(e)]
                    if e[ax]:
                        f = list(e)
                        f[ax] -= 1
                        val = val + e[ax] * cur[tuple(f)]
                    new[t, u, v] = val
        cur = new
    return cur


def _pair_blocks(mol, atoms, xyz, omega, size):
    """Every shell pair's Cartesian integral block at every point, in chunks of
    primitive pairs: (la, lb, i, j, A) with i, j the shells of the chunk's
    rows and A {(a, b): (rows, P)}."""
    P = xyz.shape[0]
    host = atoms.detach().cpu().numpy()
    for la in range(4):
        for lb in range(la + 1):
            rows = []
            for i, si in enumerate(mol.shells):
                for j, sj in enumerate(mol.shells):
                    if si.l != la or sj.l != lb or (la == lb and j > i):
                        continue
                    r2 = float(((host[si.atom] - host[sj.atom]) ** 2).sum())
                    for a, ca in zip(si.exps, si.coeffs[:, 0]):
                        for b, cb in zip(sj.exps, sj.coeffs[:, 0]):
                            if abs(ca * cb) * math.exp(-a * b / (a + b) * r2) > 1e-17:
                                rows.append((i, j, si.atom, sj.atom, a, b, ca * cb))
            step = max(1, size // P)
            for r0 in range(0, len(rows), step):
                part = rows[r0:r0 + step]
                idx = torch.tensor([r[:4] for r in part], device=xyz.device)
                a, b, cc = torch.tensor([r[4:] for r in part], dtype=torch.float64,
                                        device=xyz.device).T
                A, B = atoms[idx[:, 2]], atoms[idx[:, 3]]
                p = a + b
                C = (a[:, None] * A + b[:, None] * B) / p[:, None]
                pref = 2.0 * math.pi / p * cc * torch.exp(-a * b / p * ((A - B) ** 2).sum(dim=1))
                E = [_hermite(la, lb, p, C[:, x] - A[:, x], C[:, x] - B[:, x]) for x in range(3)]
                th = torch.ones_like(p) if omega == 0 else omega ** 2 / (omega ** 2 + p)
                alpha = (p * th)[:, None]
                X, Y, Z = (C[:, x, None] - xyz[None, :, x] for x in range(3))
                F = _boys(alpha * (X * X + Y * Y + Z * Z), la + lb)
                R = _hermite_coulomb(la + lb, F, alpha, X, Y, Z)
                pref = pref * torch.sqrt(th)
                blk = {}
                for ka, ea in enumerate(_CART[la]):
                    for kb, eb in enumerate(_CART[lb]):
                        s = 0.0
                        for t in range(ea[0] + eb[0] + 1):
                            for u in range(ea[1] + eb[1] + 1):
                                for v in range(ea[2] + eb[2] + 1):
                                    c = (pref * E[0][ea[0], eb[0], t] * E[1][ea[1], eb[1], u]
                                         * E[2][ea[2], eb[2], v])
                                    s = s + c[:, None] * R[t, u, v]
                        blk[ka, kb] = s
                yield la, lb, idx[:, 0], idx[:, 1], blk


def _solid_matrix(l, device):
    m = torch.zeros(2 * l + 1, len(_CART[l]), dtype=torch.float64, device=device)
    for row, poly in enumerate(_SOLID[l]):
        for e, c in poly.items():
            m[row, _CART[l].index(e)] = c
    return m


def _to_cart(mol, F):
    """(nshell, ncart(l), P) per l of spherical F (nao, P); rows of shells of
    another l are unused."""
    loc = mol.ao_loc_nr()
    out = []
    for l in range(4):
        m = _solid_matrix(l, F.device)
        out.append(torch.stack([m.T @ F[loc[i]:loc[i + 1]] if sh.l == l
                                else F.new_zeros(len(_CART[l]), F.shape[1])
                                for i, sh in enumerate(mol.shells)])
                   if any(sh.l == l for sh in mol.shells) else None)
    return out


def _k_exact(mol, xyz, w, D, omega):
    atoms = torch.as_tensor(mol.atom_coords(), device=xyz.device)
    X = _ao(mol, xyz, atoms)
    Fc = _to_cart(mol, D.T @ X)
    Gc = [None if f is None else torch.zeros_like(f) for f in Fc]
    for la, lb, i, j, blk in _pair_blocks(mol, atoms, xyz, omega, 1 << 21):
        off = (i != j).to(torch.float64)[:, None]
        for (a, b), s in blk.items():
            Gc[la][:, a].index_add_(0, i, s * Fc[lb][j, b])
            Gc[lb][:, b].index_add_(0, j, s * off * Fc[la][i, a])
    G = torch.cat([_solid_matrix(sh.l, xyz.device) @ Gc[sh.l][n]
                   for n, sh in enumerate(mol.shells)])
    return (X * w) @ G.T


def _grad_exact(mol, xyz, w, D, omega):
    """d/dR of E = -1/4 sum_g w F A F, F = D X, by reverse differentiation."""
    atoms = torch.as_tensor(mol.atom_coords(), device=xyz.device).requires_grad_()
    F = D @ _ao(mol, xyz, atoms)
    leaf = F.detach().requires_grad_()
    for la, lb, i, j, blk in _pair_blocks(mol, atoms, xyz, omega, 1 << 19):
        Fc = _to_cart(mol, leaf)
        fac = torch.where(i != j, 2.0, 1.0).to(torch.float64)[:, None]
        e = sum((s * Fc[la][i, a] * Fc[lb][j, b]) for (a, b), s in blk.items())
        (-0.25 * (e * fac * w).sum()).backward()
    (F * leaf.grad).sum().backward()
    return atoms.grad.cpu().numpy()


def _gga_density(X, D):
    T = D @ X[0]
    rho = torch.empty(5, X.shape[2], dtype=torch.float64, device=X.device)
    rho[0] = (T * X[0]).sum(dim=0)
    rho[4] = 0.0
    for d in range(1, 4):
        rho[d] = 2.0 * (T * X[d]).sum(dim=0)
        rho[4] += 0.5 * ((D @ X[d]) * X[d]).sum(dim=0)
    return rho


def _xc_exact(mol, xyz, w, D, xctype):
    X = _ao(mol, xyz, torch.as_tensor(mol.atom_coords(), device=xyz.device), deriv=True)
    rho = _gga_density(X, D)
    exc, vrho, vsigma, vtau = (None if v is None else torch.as_tensor(v, device=xyz.device)
                               for v in _Functional(xctype).eval(rho.cpu().numpy()))
    nelec, energy = float((rho[0] * w).sum()), float((rho[0] * w * exc).sum())
    G = 0.5 * vrho * X[0] + 2.0 * vsigma * (rho[1:4, None] * X[1:]).sum(dim=0)
    V = (X[0] * w) @ G.T
    V = V + V.T
    if vtau is not None:
        for d in range(1, 4):
            V += (X[d] * (0.5 * w * vtau)) @ X[d].T
    return nelec, energy, V.cpu().numpy()


def _vv10_exact(mol, xyz, w, D):
    b, c = NLC_PARS
    X = _ao(mol, xyz, torch.as_tensor(mol.atom_coords(), device=xyz.device), deriv=True)
    rho_all = _gga_density(X, D)
    ok = rho_all[0] >= 1e-8
    rho, wk, pos = rho_all[:, ok], w[ok], xyz[ok]
    R, S = rho[0], (rho[1:4] ** 2).sum(dim=0)
    w2 = c * (S / (R * R)) ** 2
    w0 = torch.sqrt(w2 + 4.0 * math.pi / 3.0 * R)
    kap = b * 1.5 * math.pi * (9.0 * math.pi) ** (-1.0 / 6.0) * R ** (1.0 / 6.0)
    beta = (3.0 / (b * b)) ** 0.75 / 32.0
    q = R * wk
    F, U, W = (torch.zeros_like(R) for _ in range(3))
    step = max(1, (1 << 23) // max(1, len(R)))
    for i in range(0, len(R), step):
        k = slice(i, i + step)
        r2 = ((pos[k, None, 0] - pos[None, :, 0]) ** 2 + (pos[k, None, 1] - pos[None, :, 1]) ** 2
              + (pos[k, None, 2] - pos[None, :, 2]) ** 2)
        g = r2 * w0[k, None] + kap[k, None]
        gp = r2 * w0 + kap
        T = q / (g * gp * (g + gp))
        F[k] = -1.5 * T.sum(dim=1)
        T = T * (1.0 / g + 1.0 / (g + gp))
        U[k], W[k] = T.sum(dim=1), (T * r2).sum(dim=1)
    dw_dr = (2.0 * math.pi / 3.0 - 2.0 * w2 / R) / w0
    dw_ds = w2 / (S * w0)
    exc = beta + 0.5 * F
    v_r = beta + F + 1.5 * (U * kap / 6.0 + W * R * dw_dr)
    v_s = 1.5 * W * R * dw_ds
    nelec = float((rho_all[0] * w).sum())
    energy = float((q * exc).sum())
    Xk = X[:, :, ok]
    G = 0.5 * v_r * Xk[0] + 2.0 * v_s * (rho[1:4, None] * Xk[1:]).sum(dim=0)
    V = (Xk[0] * wk) @ G.T
    return nelec, energy, (V + V.T).cpu().numpy()


def exact(case, seed):
    kind = case['kind']
    if kind in ('batch', 'fock'):
        return None
    mol = _molecule(case)
    points = _points(mol, case['level'])
    nprim = sum(sh.nprim * (sh.l + 1) ** 2 for sh in mol.shells)
    # integrals of every primitive pair at every point: some ten seconds
    if kind not in ('xc', 'vv10') and nprim ** 2 * points * (1 + (kind == 'grad') * 19) > 4e10:
        return None
    if kind in ('xc', 'vv10') and points * mol.nao > 2.5e8:
        return None
    g = _grid(case, case['level'])
    dev = torch.device('cuda' if torch.cuda.is_available() else 'cpu')
    xyz, w = torch.as_tensor(g.coords, device=dev), torch.as_tensor(g.weights, device=dev)
    D = torch.as_tensor(_density(mol, seed), device=dev)
    if kind == 'xc':
        return _xc_exact(mol, xyz, w, D, case['xctype'])
    if kind == 'vv10':
        return _vv10_exact(mol, xyz, w, D)
    if kind == 'grad':
        return _grad_exact(mol, xyz, w, D, case['omega'])
    if kind == 'k1':
        return _k_exact(mol, xyz, w, D, case['omega'])
    return torch.stack([_k_exact(mol, xyz, w, D, om) for om in OMEGAS])
