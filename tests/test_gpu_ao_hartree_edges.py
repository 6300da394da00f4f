"""AO values and gradients and the Hartree potential where their kernels can go
wrong: grids of one point, around a block of 32 and ragged, points on a nucleus
and out to 60 bohr, where every exponential has underflowed; class pair counts
that are no multiple of a chunk (a dimer has 1 to 91 pairs a class).  Against
the FP64 oracle, to the bounds of the other tests of the same quantities:
1e-13 of the largest AO value, 1e-12 (FP64) and 2e-6 (FP32) of the largest
potential."""
import numpy as np
import pytest

import oracle
from helpers import density, dimer

pytestmark = pytest.mark.gpu


def _points(mol, n):
    rng = np.random.default_rng(n)
    nuc = mol.atom_coords()
    m = max(n - len(nuc), 0)
    d = rng.normal(size=(m, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    r = np.exp(rng.uniform(np.log(1e-4), np.log(60.0), m))
    return np.concatenate([nuc, nuc[rng.integers(len(nuc), size=m)] + r[:, None] * d])[:n]


@pytest.mark.parametrize('n', [1, 31, 33, 1057])
@pytest.mark.parametrize('basis', ['synthetic-svp', 'synthetic-tzvp'])
def test_ao_and_hartree_on_edge_grids(basis, n):
    import torch

    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    mol = dimer(basis)
    # the oracle's frame: a shifted one rounds every coordinate anew, which next
    # to a nucleus moves a tight gradient by 1e-12 of its largest value
    eng = CosxEngine(mol, origin=np.zeros(3))
    pts = _points(mol, n)
    c = eng.relative(pts)
    ref = oracle.ao_eval_deriv1(mol, pts).transpose(0, 2, 1)
    X1 = eng.ao_eval_deriv1(c).cpu().numpy()
    assert np.all(X1[:, :, n:] == 0.0)
    for d in range(4):
        assert np.abs(X1[d, :, :n] - ref[d]).max() < 1e-13 * np.abs(ref[d]).max(), d
    X = eng.ao_eval(c).cpu().numpy()
    assert np.abs(X[:, :n] - ref[0]).max() < 1e-13 * np.abs(ref[0]).max()
    dm = density(mol.nao, 10, 4)
    d = torch.as_tensor(dm, device='cuda')
    v = oracle.hartree(mol, pts, dm)
    for fp64, tol in ((True, 1e-12), (False, 2e-6)):
        got = eng.hartree(c, d, tol=0.0, fp64=fp64).cpu().numpy()
        assert np.abs(got - v).max() < tol * np.abs(v).max(), fp64
