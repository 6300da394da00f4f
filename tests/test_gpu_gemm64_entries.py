"""What the splits behind the FP64 products promise for a single entry.  With W =
7 S bits (S = 10 digits for F, 9 for K) below 2^e and 2^f, the powers of two above
the largest entries of the row and the column (X_max >= 2^(e-1), Q_max >=
2^(f-1)): each operand is rounded to a multiple of 2^(e - W + 1), within 2^(2 - W
- 1) X_max; the dropped digit products, (2 S - 1 - l) of at most 2^12 at each
level l >= S, of scale 2^(e + f - 2 W + 2 + 7 (2 S - 2 - l)), sum to at most
9.07 2^(e + f + 7 S - 2 W) (S = 10: 2^-64.8, S = 9: 2^-57.9 X_max Q_max).  So a
term of the product is within TERM[S] X_max Q_max whatever its own size, and the
sum is rounded once.  Against extended precision on the host, entries from the
maxima down to 10^-30 of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TERM = {10: 2.0 ** -64.6, 9: 2.0 ** -57.7}


def _product(a, b):
    return np.stack([(r[:, None].astype(np.longdouble) * b.astype(np.longdouble)).sum(0)
                     for r in a])


def _check(got, a, b, digits):
    ref = _product(a, b)
    top = np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :]
    err = np.abs(got.astype(np.longdouble) - ref)
    assert np.all(err <= a.shape[1] * TERM[digits] * top + 2.0 ** -53 * np.abs(ref) + 1e-300)


@pytest.mark.parametrize('spread', [0.0, 8.0, 30.0])
def test_entries(spread):
    import torch

    from helpers import dimer
    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    mol = dimer()
    eng = CosxEngine(mol)
    rng = np.random.default_rng(int(spread))

    def matrix(*shape):
        return rng.normal(size=shape) * 10.0 ** rng.uniform(-spread, 0.0, shape)

    X, Q, G, w = matrix(mol.nao, 320), matrix(mol.nao, mol.nao), matrix(mol.nao, 320), \
        rng.uniform(0.1, 2.0, 320)
    dev = [torch.as_tensor(t, device='cuda') for t in (X, Q, G, w)]
    _check(eng.gemm64_f(dev[0], dev[1]).cpu().numpy().T, X.T.copy(), Q, 10)
    wg = (dev[2] * dev[3]).cpu().numpy()
    _check(eng.gemm64_k(dev[0], dev[2], dev[3]).cpu().numpy(), X, wg.T.copy(), 9)
