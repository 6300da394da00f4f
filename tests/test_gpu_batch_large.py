"""Batched K builds with a molecule that fills the device on its own (more than
ten 64-point blocks an SM): it runs its own class launches inside the batch.  K
bitwise its single build's, with one omega and two, again on a second run (block
order learnt), and with either molecule left out."""
import pytest

from helpers import density, dimer, grid_subset, waters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('omegas', [(0.0, 0.3), (0.3,)])
def test_large_and_small_molecules_in_one_batch(omegas):
    import torch

    from pyscf_wb97mv_fast_gb300.cosx import CosxBatch, CosxEngine
    mols = [dimer('synthetic-svp'), waters(24, 9.6, 5)]
    engines, grids, dms, ref = [], [], [], []
    for i, mol in enumerate(mols):
        c, w = grid_subset(mol, 0, None)
        assert (len(c) > 640 * torch.cuda.get_device_properties(0).multi_processor_count) == (i == 1)
        eng, alone = CosxEngine(mol), CosxEngine(mol)
        cd, wd = eng.relative(c), torch.as_tensor(w, device='cuda')
        dm = torch.as_tensor(density(mol.nao, 5 * (1 + 20 * i), i), device='cuda')
        engines.append(eng)
        grids.append((cd, wd))
        dms.append(dm)
        ref.append(alone.get_k_multi(cd, wd, dm, omegas, tile_tol=1e-11).clone())
    b = CosxBatch(engines, grids, omegas, tile_tol=1e-11)
    for qd in ([0, 1], [0, 1], [0, None], [None, 1]):
        Ks = b.run([None if q is None else dms[q] for q in qd], stats=True)
        for K, q, r in zip(Ks, qd, ref):
            assert (K is None) == (q is None)
            assert K is None or torch.equal(K, r)
    b.close()
