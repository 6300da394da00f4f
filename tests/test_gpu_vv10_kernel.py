"""A caller's own double sum in the VV10 flows: it is given q, W0 and kappa in
FP64 (the library's own sum works on FP32 values), and an FP64 one is not
limited by a rounding before it.  And AO values of any padding in the FP64 flow."""
import types

import numpy as np
import pytest

from helpers import density, dimer, grid_subset

pytestmark = pytest.mark.gpu

PARS = (6.0, 0.01)


class Fp64Sum:
    """F = -1.5 sum_j q_j / (g g' (g + g')), U and W its weighted forms, in
    FP64; records what it was given."""

    def __init__(self):
        self.seen = []

    def kernel_sum(self, coords, q, W0, kappa):
        import torch
        self.seen.append((coords, q, W0, kappa))
        r = coords.to(torch.float64)
        R2 = ((r[:, None, :] - r[None, :, :]) ** 2).sum(-1)
        a, b, k = (x.to(torch.float64) for x in (q, W0, kappa))
        g = R2 * b[:, None] + k[:, None]
        gp = R2 * b[None, :] + k[None, :]
        T = a[None, :] / (g * gp * (g + gp))
        Tu = T * (1.0 / g + 1.0 / (g + gp))
        return -1.5 * T.sum(1), Tu.sum(1), (Tu * R2).sum(1)


@pytest.fixture(scope='module')
def case():
    import torch

    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine
    from pyscf_wb97mv_fast_gb300.scf import DeviceGrid
    mol = dimer()
    coords, weights = grid_subset(mol, 1, 1500, 3)
    eng = CosxEngine(mol)
    g = DeviceGrid(eng, types.SimpleNamespace(coords=coords, weights=weights), deriv=1)
    dm = density(mol.nao, 10, 3)
    return mol, coords, weights, eng, g, torch.as_tensor(dm, device=eng.device), dm


def _check_inputs(eng, g, dm, seen):
    import torch

    from pyscf_wb97mv_fast_gb300.gpu.vv10 import THRESH, vv10_pointwise
    X = g.X[:, :, :g.n]
    T = dm @ X[0]
    rho = (T * X[0]).sum(0)
    grad = 2.0 * torch.einsum('mp,dmp->dp', T, X[1:])
    ind = rho >= THRESH
    ref = vv10_pointwise(rho[ind], grad[:, ind], g.weights[ind], PARS)[:3]
    for got, want in zip(seen[1:], ref):
        assert got.dtype == torch.float64 and got.shape == want.shape
        # sums of nao products in FP64 on either side
        assert float(((got - want) / want).abs().max()) < 1e-10


def test_energy_fock_with_an_fp64_sum(case):
    from pyscf_wb97mv_fast_gb300.gpu.vv10 import vv10_energy_fock
    mol, coords, weights, eng, g, dm, _ = case
    k = Fp64Sum()
    e, v = vv10_energy_fock(eng, g, dm, PARS, kernel=k)
    _check_inputs(eng, g, dm, k.seen[0])
    e0, v0 = vv10_energy_fock(eng, g, dm, PARS)
    assert abs(float(e - e0)) < 1e-6 * abs(float(e0))
    assert float((v - v0).abs().max()) < 1e-5 * float(v0.abs().max())


def test_nlc_vxc_with_an_fp64_sum(case):
    from pyscf_wb97mv_fast_gb300.gpu.vv10 import Vv10Context, gpu_nr_nlc_vxc
    mol, coords, weights, eng, g, dm, dm_h = case
    ni = types.SimpleNamespace(nlc_coeff=lambda xc: ((PARS, 1.0),))
    grids = types.SimpleNamespace(coords=coords, weights=weights)
    ctx = Vv10Context(mol)
    n0, e0, v0 = gpu_nr_nlc_vxc(ctx, ni, mol, grids, 'vv10', dm_h)
    ctx.kernel = Fp64Sum()
    n1, e1, v1 = gpu_nr_nlc_vxc(ctx, ni, mol, grids, 'vv10', dm_h)
    _check_inputs(eng, g, dm, ctx.kernel.seen[0])
    assert n1 == n0 and abs(e1 - e0) < 1e-6 * abs(e0)
    assert np.max(np.abs(v1 - v0)) < 1e-5 * np.abs(v0).max()


@pytest.mark.parametrize('ld', [1500, 1501, 1536, 2048])
def test_fp64_flow_takes_any_padding(case, ld):
    """The FP64 flow on AO values padded to another length than the library's:
    the same numbers."""
    import torch

    from pyscf_wb97mv_fast_gb300.gpu.vv10 import vv10_energy_fock
    mol, coords, weights, eng, g, dm, _ = case
    e0, v0 = vv10_energy_fock(eng, g, dm, PARS)
    X = torch.zeros((4, mol.nao, ld), dtype=torch.float64, device=eng.device)
    X[:, :, :g.n] = g.X[:, :, :g.n]
    other = types.SimpleNamespace(n=g.n, coords=g.coords, weights=g.weights, X=X)
    e, v = vv10_energy_fock(eng, other, dm, PARS)
    assert torch.equal(e, e0) and torch.equal(v, v0)
