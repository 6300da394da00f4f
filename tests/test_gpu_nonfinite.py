"""A NaN or an infinity in a K build's operands shows in what it enters: the
split products give NaN for the rows and columns that hold one (and the others
bit for bit as without it), and the screen drops no pair on a bound that is no
number.  So a density that has diverged, or a tensor-core F product whose wait
gave up (NaN in its 128 points), cannot end as a finite K that lacks points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VALUES = [float('nan'), float('inf'), -float('inf')]


def _setup(n):
    import torch

    from helpers import density, dimer
    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    mol = dimer('synthetic-svp')
    eng = CosxEngine(mol)
    rng = np.random.default_rng(n)
    pts = mol.atom_coords()[rng.integers(mol.natm, size=n)] + rng.normal(size=(n, 3))
    c = eng.relative(pts)
    w = torch.as_tensor(rng.uniform(0.1, 1.0, n), device=eng.device)
    dm = torch.as_tensor(density(mol.nao, 10, 3), device=eng.device)
    return eng, c, w, dm


@pytest.mark.parametrize('value', VALUES)
@pytest.mark.parametrize('engine', ['library', 'tc'])
@pytest.mark.parametrize('fp64', [False, True])
def test_f_product(engine, value, fp64):
    import torch

    from pyscf_wb97mv_fast_gb300 import cosx
    eng, c, w, dm = _setup(300)
    X = eng.ao_eval(c)
    bad = dm.clone()
    bad[5, 7] = value
    prev = cosx.set_f_engine(engine)
    try:
        ref, F = (eng.ozaki_f(X, d, fp64=fp64) for d in (dm, bad))
    finally:
        cosx.set_f_engine(prev)
    rows = [i for i in range(eng.nao) if i != 7]
    assert torch.equal(F[rows], ref[rows])
    assert bool(torch.isnan(F[7, :300]).all())


@pytest.mark.parametrize('value', VALUES)
@pytest.mark.parametrize('n', [300, 2100])
def test_k_product(n, value):
    import torch
    eng, c, w, dm = _setup(n)
    X = eng.ao_eval(c)
    for G in (eng.ozaki_f(X, dm), eng.ozaki_f(X, dm, fp64=True)):
        bad = G.clone()
        bad[11, n - 1] = value
        ref, K = (eng.ozaki_k(X, g, w) for g in (G, bad))
        cols = [i for i in range(eng.nao) if i != 11]
        assert torch.equal(K[:, cols], ref[:, cols])
        assert bool(torch.isnan(K[:, 11]).all())


@pytest.mark.parametrize('omegas', [(0.0,), (0.0, 0.3)])
def test_g_and_k_of_a_point_without_f(omegas):
    import torch
    eng, c, w, dm = _setup(300)
    F = eng.ozaki_f(eng.ao_eval(c), dm)
    F[:, 200] = float('nan')
    G = eng.g_multi(c, w, F, omegas, tile_tol=1e-8)
    assert bool(torch.isnan(G[:, :, 200]).all())
    others = [i for i in range(300) if i != 200]
    assert bool(torch.isfinite(G[:, :, others]).all())
    bad = dm.clone()
    bad[5, 7] = float('nan')
    K = eng.get_k_multi(c, w, bad, omegas, tile_tol=1e-8, stats=False)
    assert bool(torch.isnan(K).any())
    assert bool(torch.isnan(eng.get_k_fp64(c, w, bad, omegas, tile_tol=1e-8)).any())
