"""A captured K build replays on buffers of its own: direct builds on the same
engine between the replays, on smaller and larger grids, and calls that make the
engine's workspace grow, change neither its result nor theirs."""
import numpy as np
import pytest

from helpers import density, dimer

pytestmark = pytest.mark.gpu


def _grid(eng, n, seed):
    import torch
    rng = np.random.default_rng(seed)
    pts = eng.mol.atom_coords()[rng.integers(eng.mol.natm, size=n)] + rng.normal(size=(n, 3))
    return eng.relative(pts), torch.as_tensor(rng.uniform(0.1, 1.0, n), device=eng.device)


@pytest.mark.parametrize('between', ['smaller', 'larger', 'workspace'])
@pytest.mark.parametrize('omegas', [(0.0,), (0.0, 0.3)])
def test_replays_after_other_builds(omegas, between):
    import torch

    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    mol = dimer()
    fresh, eng = CosxEngine(mol), CosxEngine(mol)
    dms = [torch.as_tensor(density(mol.nao, 10, k), device=eng.device) for k in range(3)]

    def direct(e, grid, dm):
        K = e.get_k_multi(*grid, dm, omegas, tile_tol=1e-11)
        return (K + K.transpose(1, 2)) * 0.5

    grid = _grid(eng, 5000, 1)
    want = [direct(fresh, grid, d) for d in dms]
    graph = eng.capture_k_multi(*grid, omegas, tile_tol=1e-11)
    other = _grid(eng, dict(smaller=1000, larger=20000, workspace=5000)[between], 2)
    want_other = direct(fresh, other, dms[0])
    for _ in range(2):
        for d, w in zip(dms, want):
            assert torch.equal(graph.run(d), w)
            if between == 'workspace':
                eng.gemm64_f(torch.randn((mol.nao, 64000), dtype=torch.float64,
                                         device=eng.device), d)
                # whatever was given back is taken and overwritten
                junk = [torch.full((1 << 20,), float('nan'), device=eng.device)
                        for _ in range(64)]
                del junk
            else:
                assert torch.equal(direct(eng, other, dms[0]), want_other)
    assert torch.equal(direct(eng, grid, dms[1]), want[1])
