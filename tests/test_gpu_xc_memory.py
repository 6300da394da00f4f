"""tile_pts bounds the memory of the semilocal flow: tiles that it limits come
one after another (no AO values of another tile alive when a tile's are made),
and the look-ahead of smaller tiles holds two at a time.  The result does not
depend on it."""
import types
import weakref

import numpy as np
import pytest

from helpers import ToyFunctional, ToyNumInt, density, dimer

pytestmark = pytest.mark.gpu


def _run(mol, n, tile_pts):
    from pyscf_wb97mv_fast_gb300.gpu.xc import XcContext, gpu_nr_rks
    rng = np.random.default_rng(n)
    coords = mol.atom_coords()[rng.integers(mol.natm, size=n)] + rng.normal(size=(n, 3))
    grids = types.SimpleNamespace(coords=coords, weights=rng.uniform(1e-3, 1e-2, n))
    ctx = XcContext(mol, functional_factory=lambda xc, ni: ToyFunctional('MGGA'),
                    tile_pts=tile_pts)
    eng = ctx.build()
    made, alive = [], []
    inner = eng.ao_eval_deriv1

    def ao_eval_deriv1(c, *a, **k):
        alive.append(sum(r() is not None for r in made))
        X = inner(c, *a, **k)
        made.append(weakref.ref(X))
        return X

    eng.ao_eval_deriv1 = ao_eval_deriv1
    out = gpu_nr_rks(ctx, ToyNumInt('MGGA'), mol, grids, 'toy', density(mol.nao, 10, 3))
    return alive, out


@pytest.mark.parametrize('n,tile_pts,most', [(9000, 2048, 0), (140000, 40000, 0),
                                             (140000, 50000, 0), (140000, 1 << 20, 1)])
def test_tiles_held(n, tile_pts, most):
    mol = dimer()
    alive, (nelec, exc, v) = _run(mol, n, tile_pts)
    assert len(alive) > 1 and max(alive) == most
    _, (nelec1, exc1, v1) = _run(mol, n, n + 1 if n < 1 << 16 else n)
    assert abs(nelec - nelec1) <= 1e-12 * abs(nelec1)
    assert abs(exc - exc1) <= 1e-11 * abs(exc1)
    assert np.max(np.abs(v - v1)) <= 1e-10 * np.abs(v1).max()
