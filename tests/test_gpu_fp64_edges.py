"""The FP64 class and gradient kernels where they can go wrong: ragged last
blocks, grids of fewer blocks than warps, points on a nucleus (T = 0), around
the switch of the Boys forms (T = 36) and far out.  K against the FP64 oracle
to the 1e-11 relative of the FP64 tests; the gradient is a sum over points, so
the gradient of a grid is that of its parts to FP64 summation error (1e-12)."""
import numpy as np
import pytest

import oracle
from helpers import density, dimer

pytestmark = pytest.mark.gpu


def _points(mol, n, seed):
    """n points: nuclei first, then random directions at radii from 1e-4 to 60
    bohr (log-spaced), which sweeps T = p r^2 through 36 for every exponent."""
    rng = np.random.default_rng(seed)
    nuc = mol.atom_coords()
    m = max(n - len(nuc), 0)
    d = rng.normal(size=(m, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    r = np.exp(rng.uniform(np.log(1e-4), np.log(60.0), m))
    pts = np.concatenate([nuc, nuc[rng.integers(len(nuc), size=m)] + r[:, None] * d])[:n]
    return pts, rng.uniform(0.1, 1.0, n)


@pytest.mark.parametrize('basis,n', [('synthetic-svp', 1), ('synthetic-svp', 31),
                                     ('synthetic-svp', 33), ('synthetic-svp', 1025),
                                     ('synthetic-tzvp', 33), ('synthetic-tzvp', 449)])
def test_fp64_k_and_gradient_on_edge_grids(basis, n):
    import torch

    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    mol = dimer(basis)
    pts, w = _points(mol, n, n)
    dm = density(mol.nao, 10, 3)
    eng = CosxEngine(mol)
    c = eng.relative(pts)
    wt = torch.as_tensor(w, device=eng.device)
    qd = torch.as_tensor(dm, device=eng.device)
    K = eng.get_k_fp64(c, wt, qd, (0.0, 0.3), tile_tol=0.0)
    K = ((K + K.transpose(1, 2)) * 0.5).cpu().numpy()
    for j, om in enumerate((0.0, 0.3)):
        Kref = oracle.cosx_k(mol, pts, w, dm, om)
        assert np.max(np.abs(K[j] - Kref)) < 1e-11 * np.abs(Kref).max(), om
        g = eng.k_grad(c, wt, dm, om)
        h = max(1, n // 3)
        parts = sum(eng.k_grad(c[s].contiguous(), wt[s].contiguous(), dm, om)
                    for s in (slice(0, h), slice(h, n)) if s.stop > s.start)
        assert np.max(np.abs(g - parts)) < 1e-12 * np.abs(g).max(), om
