"""The XC and GGA point kernels' vector and scalar forms: arrays that start off a
16-byte boundary give bitwise what aligned ones do, over ragged grids and AO
counts that are no multiple of 8 or 64; and the density against FP64 sums.  Its
products and sums of 8 AOs are FP32: 2^-20 of the sum of the terms' magnitudes
(eight roundings of 2^-24 each in a group, two more for the factors)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _off(t):
    """A copy of t one element past an aligned start."""
    import torch
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    v = buf[1:].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize('basis,n', [('synthetic-svp', 1), ('synthetic-svp', 63),
                                     ('synthetic-tzvp', 65), ('synthetic-tzvp', 700)])
@pytest.mark.parametrize('mgga', [False, True])
def test_unaligned_arrays(basis, n, mgga):
    import torch

    from helpers import dimer
    from pyscf_wb97mv_fast_gb300.cosx import CosxEngine, round32
    mol = dimer(basis)
    eng = CosxEngine(mol)
    g = torch.Generator(device='cuda').manual_seed(n)
    ld, nao = round32(n), mol.nao

    def rand(*shape):
        return torch.randn(*shape, dtype=torch.float64, device='cuda', generator=g)

    X, v = rand(4, nao, ld), rand(5, ld)
    T = rand(4 if mgga else 1, nao, ld).to(torch.float32)
    rho = eng.xc_rho(X, T, n, mgga)
    assert torch.equal(eng.xc_rho(_off(X), _off(T), n, mgga), rho)
    X32, T64 = X.to(torch.float32).to(torch.float64), T.to(torch.float64)
    terms = [T64[0] * X32[d] for d in range(4)]
    if mgga:
        terms.append((T64[1:] * X32[1:]).sum(0))
    for k, t in enumerate(terms):
        f = 1.0 if k == 0 else 0.5 if k == 4 else 2.0
        mag = t.abs().sum(0) if k < 4 else (T64[1:] * X32[1:]).abs().sum((0, 1))
        err = (rho[k, :n] - f * t.sum(0)[:n]).abs()
        assert bool((err <= f * 2.0 ** -20 * mag[:n]).all()), k
    assert bool((rho[:, n:] == 0).all())
    G = eng.xc_aow(X, v, n, mgga)
    assert torch.equal(eng.xc_aow(_off(X), _off(v), n, mgga), G)
    for out in (None, torch.float32):
        A = eng.gga_aow(X, v[:4].contiguous(), n, out)
        assert torch.equal(eng.gga_aow(_off(X), _off(v[:4]), n, out), A)
