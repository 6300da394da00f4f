"""The FP64 products on the tensor cores (wb_cosx_gemm64_f / _k) and the FP64
GGA kernels, where they can go wrong: AO counts that are no multiple of 8,
level sums cut in pieces (nao > 455), ragged grids, several point tiles and
chunk groups, rows that span the exponent range, infinities and NaN.

Reference: the same product in twice FP64 (exact products by fma splitting is
not at hand in torch, so both operands are cut into 26-bit halves whose FP64
products are exact and summed in groups).  Bound: the error is at most that of
the FP64 GEMM plus 2^-52 of the result in the 2-norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(name):
    from helpers import dimer, waters
    from pyscf_wb97mv_fast_gb300.basis import Molecule
    from pyscf_wb97mv_fast_gb300.systems import alkane
    return {'dimer': dimer, 'waters4': lambda: waters(4, 6.0, 3),
            'ethane': lambda: Molecule.build(alkane(2), 'synthetic-tzvp'),
            'undecane': lambda: Molecule.build(alkane(11), 'synthetic-tzvp')}[name]()


def _wide(a, b):
    """a @ b with a, b cut into three 18-bit pieces (exact products, FP64 sums
    of pieces of like size): error well below one FP64 GEMM's."""
    import torch

    def cut(x):
        out = []
        for _ in range(2):
            m, e = torch.frexp(x.abs().amax())
            s = torch.ldexp(torch.tensor(1.0, dtype=x.dtype, device=x.device), e - 18)
            h = torch.round(x / s) * s
            out.append(h)
            x = x - h
        return out + [x]

    A, B = cut(a), cut(b)
    acc = [A[i] @ B[j] for i in range(3) for j in range(3)]
    return sum(sorted(acc, key=lambda t: float(t.abs().max())))


@pytest.mark.parametrize('name,n', [('dimer', 1), ('dimer', 33), ('waters4', 4000),
                                    ('ethane', 511), ('ethane', 70001),
                                    ('undecane', 1500)])
def test_products_as_accurate_as_fp64(name, n):
    import torch

    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine, round32
    mol = _case(name)
    eng = CosxEngine(mol)
    rng = np.random.default_rng(n)
    nuc = mol.atom_coords()
    r = np.exp(rng.uniform(np.log(1e-3), np.log(12.0), (n, 1)))
    d = rng.normal(size=(n, 3))
    pts = nuc[rng.integers(len(nuc), size=n)] + r * d / np.linalg.norm(d, axis=1)[:, None]
    X = eng.ao_eval(eng.relative(pts))
    c = torch.as_tensor(rng.normal(size=(mol.nao, 7)), device='cuda')
    D = c @ c.T
    ld = round32(n)
    F = eng.gemm64_f(X, D)
    ref = _wide(D.T.contiguous(), X)
    own = (D.T @ X - ref).norm()
    assert float((F - ref).norm()) <= float(own) + 2.0 ** -52 * float(ref.norm())
    w = torch.as_tensor(rng.uniform(0.01, 2.0, n), device='cuda')
    G = torch.randn(X.shape, dtype=torch.float64, device='cuda')
    K = eng.gemm64_k(X, G, w)
    wg = torch.zeros_like(G)
    wg[:, :n] = G[:, :n] * w
    ref = _wide(X, wg.T.contiguous())
    own = (X @ wg.T - ref).norm()
    assert float((K - ref).norm()) <= float(own) + 2.0 ** -52 * float(ref.norm())
    assert X.shape[1] == ld


def test_extreme_values():
    """Rows over the whole exponent range scale exactly; infinities and NaN
    give NaN in their row or column and leave the others alone."""
    import torch

    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    mol = _case('dimer')
    eng = CosxEngine(mol)
    nao = mol.nao
    X = torch.randn((nao, 64), dtype=torch.float64, device='cuda')
    D = torch.randn((nao, nao), dtype=torch.float64, device='cuda')
    base = eng.gemm64_f(X, D)
    # exact powers of two from their bits (torch.ldexp goes through pow)
    k = torch.linspace(-900, 900, 64, device='cuda').round().to(torch.int64)
    p2 = ((k + 1023) << 52).view(torch.float64)
    assert torch.equal(eng.gemm64_f(X * p2, D), base * p2)
    Y = X.clone()
    Y[3, 5] = float('nan')
    Y[2, 9] = float('inf')
    out = eng.gemm64_f(Y, D)
    bad = torch.zeros(64, dtype=torch.bool, device='cuda')
    bad[5] = bad[9] = True
    assert bool(torch.isnan(out[:, bad]).all())
    assert torch.equal(out[:, ~bad], base[:, ~bad])
    w = torch.ones(64, dtype=torch.float64, device='cuda')
    K = eng.gemm64_k(Y, X, w)
    assert bool(torch.isnan(K[[2, 3]]).all()) and bool(torch.isfinite(K[4:]).all())


@pytest.mark.parametrize('n', [1, 32, 45, 1000])
def test_gga_kernels(n):
    """Density, gradient and Fock-side plane against torch FP64 (sums of nao
    terms: 1e-13 of the largest), FP32 forms rounded once."""
    import torch

    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine, round32
    mol = _case('ethane')
    eng = CosxEngine(mol)
    ld = round32(n)
    X = torch.randn((4, mol.nao, ld), dtype=torch.float64, device='cuda')
    T = torch.randn((mol.nao, ld), dtype=torch.float64, device='cuda')
    for t in (T, T.to(torch.float32)):
        ref = torch.einsum('mp,dmp->dp', t.to(torch.float64), X)
        ref[1:] *= 2.0
        ref[:, n:] = 0.0
        assert float((eng.gga_rho(X, t, n) - ref).abs().max()) < 1e-13 * mol.nao
    v = torch.randn((4, ld), dtype=torch.float64, device='cuda')
    ref = torch.einsum('dp,dmp->mp', v, X)
    ref[:, n:] = 0.0
    G = eng.gga_aow(X, v, n)
    assert float((G - ref).abs().max()) < 1e-14
    assert torch.equal(eng.gga_aow(X, v, n, torch.float32), G.to(torch.float32))
