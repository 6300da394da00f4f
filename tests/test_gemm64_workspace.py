"""The 63-bit split's workspace is bounded in bytes: its point tiles and groups
of chunks shrink as the AOs grow.  On the CPU the byte count over sizes; on the
GPU both products of a size whose tiles are shrunk, against FP64 in the 2-norm
as in test_gpu_gemm64.py."""
import pytest

from pyscf_wb97mv_fast_gb300 import _native

LIMIT = 4 << 30                      # of what grows with the points of a tile


def test_bytes_are_bounded():
    get = _native.lib().wb_gemm64_workspace_bytes
    for nao in (1, 7, 48, 64, 192, 384, 442, 648, 872, 1000, 2000, 3000, 4000, 6000):
        last = 0
        for ld in (32, 1024, 65536, 65568, 131072, 400000 // 32 * 32, 4 << 20):
            b = get(nao, ld)
            digits = 18 * (nao + 7) // 8 * 8 * nao           # of the AO matrix
            assert last <= b <= LIMIT + digits + (1 << 20), (nao, ld, b)
            last = b
    # tiles of 65,536 points and 128 chunks, the measured ones, where they fit
    assert get(442, 1 << 20) == get(442, 65536)
    assert get(442, 65536) > get(442, 32768)


@pytest.mark.gpu
def test_products_in_shrunk_tiles():
    import numpy as np
    import torch

    from pyscf_wb97mv_fast_gb300.basis import Molecule
    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    from pyscf_wb97mv_fast_gb300.systems import water_cluster
    from test_gpu_gemm64 import _wide
    mol = Molecule.build(water_cluster(40, box=14.0, seed=1), 'synthetic-svp')
    n = 66000                                     # 960 AOs: tiles of 57,000 points, 78 chunks
    eng = CosxEngine(mol)
    rng = np.random.default_rng(n)
    pts = mol.atom_coords()[rng.integers(mol.natm, size=n)] + rng.normal(size=(n, 3))
    X = eng.ao_eval(eng.relative(pts))
    c = torch.as_tensor(rng.normal(size=(mol.nao, 7)), device='cuda')
    D = c @ c.T
    ref = _wide(D.T.contiguous(), X)
    own = float((D.T @ X - ref).norm())
    F = eng.gemm64_f(X, D)
    assert float((F - ref).norm()) <= own + 2.0 ** -52 * float(ref.norm())
    w = torch.as_tensor(rng.uniform(0.01, 2.0, n), device='cuda')
    wg = torch.zeros_like(F)
    wg[:, :n] = F[:, :n] * w
    ref = _wide(X, wg.T.contiguous())
    own = float((X @ wg.T - ref).norm())
    K = eng.gemm64_k(X, F, w)
    assert float((K - ref).norm()) <= own + 2.0 ** -52 * float(ref.norm())
