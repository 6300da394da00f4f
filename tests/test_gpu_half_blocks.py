"""The light classes' half blocks (two warps per 64-point block on grids of few
blocks) against whole blocks: the G of a grid's first points as a grid of their
own is that of the whole grid for every block the two share, bitwise."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('basis,n', [('synthetic-svp', 64), ('synthetic-svp', 33 + 64),
                                     ('synthetic-svp', 4096), ('synthetic-svp', 30001),
                                     ('synthetic-tzvp', 96), ('synthetic-tzvp', 5000)])
@pytest.mark.parametrize('omegas', [(0.0, 0.3), (0.0,), (0.3,)])
def test_g_of_a_small_grid_is_the_large_grids(basis, n, omegas):
    import torch

    from helpers import dimer
    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine, round32
    mol = dimer(basis)
    eng = CosxEngine(mol)
    rng = np.random.default_rng(n)
    total = 64 * 1700                       # 1,700 blocks: whole ones
    nuc = mol.atom_coords()
    pts = nuc[rng.integers(len(nuc), size=total)] + 2.0 * rng.normal(size=(total, 3))
    pts = pts[np.argsort(pts[:, 0])]        # blocks that screen
    c = eng.relative(pts)
    w = torch.as_tensor(rng.uniform(0.1, 1.0, total), device=eng.device)
    f = torch.as_tensor(rng.normal(size=(mol.nao, total)), dtype=torch.float32,
                        device=eng.device)
    big = eng.g_multi(c, w, f, omegas, tile_tol=1e-7)
    ld = round32(n)
    fs = f[:, :ld].clone()
    small = eng.g_multi(c[:n].contiguous(), w[:n].contiguous(), fs, omegas, tile_tol=1e-7)
    shared = n // 64 * 64
    assert shared and torch.equal(small[:, :, :shared], big[:, :, :shared])
