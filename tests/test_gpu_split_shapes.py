"""The 42-bit split GEMMs at the shapes where their layout changes: AO counts
that are no multiple of 8 (padded slices), grids around the 512- and 2048-point
chunks of the K product.  Against FP64 products, to the split's worst case per
term, relative to the product of the row's and the column's largest entries
(each at least half its power of two 2^e, 2^f): both operands are rounded at
2^(e - 42), which is 2 x 2^-41; the dropped digit products sum to at most
6.1 x 2^(e + f - 42) with seven 6-bit digits (levels 7 to 12, digits at most
32) and 5.1 x 2^(e + f - 42) with six 7-bit ones (levels 6 to 10, at most 64),
which is 6.1 x 2^-40; together below 2^-37."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [1, 511, 513, 2047, 2049, 6145])
@pytest.mark.parametrize('carbons', [2, 3, 8])
def test_split_products(carbons, n):
    import torch

    from pyscf_wb97mv_fast_gb300.basis import Molecule
    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    from pyscf_wb97mv_fast_gb300.systems import alkane
    mol = Molecule.build(alkane(carbons), 'synthetic-tzvp')
    eng = CosxEngine(mol)
    rng = np.random.default_rng(n)
    pts = mol.atom_coords()[rng.integers(mol.natm, size=n)] + rng.normal(size=(n, 3))
    X = eng.ao_eval(eng.relative(pts))
    c = torch.as_tensor(rng.normal(size=(mol.nao, 9)), device='cuda')
    D = c @ c.T
    ref = D.T @ X
    bound = X.abs().amax(dim=0) * D.abs().amax(dim=0)[:, None] * mol.nao * 2.0 ** -37
    assert bool(((eng.ozaki_f(X, D, fp64=True) - ref).abs() <= bound + 1e-300).all())
    w = torch.as_tensor(rng.uniform(0.1, 2.0, n), device='cuda')
    G = torch.randn(X.shape, dtype=torch.float64, device='cuda')
    for g in (G, G.to(torch.float32)):
        wg = g.to(torch.float64)[:, :n] * w
        K = eng.ozaki_k(X, g, w)
        scale = X.abs().amax(dim=1)[:, None] * wg.abs().amax(dim=1)[None, :]
        assert bool(((K - X[:, :n] @ wg.T).abs() <= scale * n * 2.0 ** -37 + 1e-300).all())
        acc = eng.ozaki_k(X, g, w, out=K.clone(), accumulate=True)
        assert float((acc - 2.0 * K).abs().max()) <= 2.0 ** -50 * float(K.abs().max())


@pytest.mark.parametrize('molecules', [28, 29])
def test_digit_forms_meet(molecules):
    """672 AOs take six 7-bit digits, 696 seven 6-bit ones: each within the
    bound above, and both engines of F bitwise equal."""
    import torch

    from pyscf_wb97mv_fast_gb300 import cosx
    from pyscf_wb97mv_fast_gb300.basis import Molecule
    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    from pyscf_wb97mv_fast_gb300.systems import water_cluster
    mol = Molecule.build(water_cluster(molecules, box=12.0, seed=1), 'synthetic-svp')
    eng = CosxEngine(mol)
    rng = np.random.default_rng(molecules)
    pts = mol.atom_coords()[rng.integers(mol.natm, size=700)] + rng.normal(size=(700, 3))
    X = eng.ao_eval(eng.relative(pts))
    c = torch.as_tensor(rng.normal(size=(mol.nao, 9)), device='cuda')
    D = c @ c.T
    bound = X.abs().amax(dim=0) * D.abs().amax(dim=0)[:, None] * mol.nao * 2.0 ** -37
    assert bool(((eng.ozaki_f(X, D, fp64=True) - D.T @ X).abs() <= bound + 1e-300).all())
    prev = cosx.set_f_engine('library')
    try:
        F = eng.ozaki_f(X, D)
        cosx.set_f_engine('tc')
        assert torch.equal(eng.ozaki_f(X, D), F)
    finally:
        cosx.set_f_engine(prev)
