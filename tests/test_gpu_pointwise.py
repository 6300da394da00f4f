"""The pointwise kernels (wb_vv10_points / _potential, wb_rsh_lda_eval) against
the same formulas in torch on the host, from the lowest densities taken to
compressed ones, with block remainders and scattered points.

Bounds, from the formulas: FP32 outputs are one rounding of an FP64 value (one
unit in the last place); FP64 sums are within 2^-46 of the sum of their terms'
magnitudes (some sixty operations of 2^-53 each); the attenuation function's
closed form sums terms up to 4 a^3 = 13.5 at a <= 1.5, a few 1e-14 of the
unattenuated exchange, and the correlation logarithms up to 30, a few 1e-16."""
import numpy as np
import pytest


def _density(n, seed):
    rng = np.random.default_rng(seed)
    return rng, 10.0 ** rng.uniform(-8.0, 3.0, n)


@pytest.mark.gpu
@pytest.mark.parametrize('n,nk', [(1, 1), (40, 0), (127, 127), (300, 128), (1000, 129)])
def test_vv10_points_and_potential(n, nk):
    import torch

    from pyscf_wb97mv_fast_gb300.gpu.vv10 import _add_potential, _points, vv10_pointwise
    rng, r = _density(n, n)
    ld = n + 5
    rho = np.zeros((4, ld))
    rho[0, :n] = r
    rho[1:, :n] = rng.normal(size=(3, n)) * r ** (4.0 / 3.0)
    coords, w = rng.normal(size=(n, 3)), rng.uniform(0.0, 1.0, n)
    ind = np.sort(rng.permutation(n)[:nk])
    F, U, W = rng.normal(size=(3, nk))
    pars, fac = (6.0, 0.01), 0.7
    host = [torch.as_tensor(x) for x in (rho, coords, w, ind, F, U, W)]
    hr, hc, hw, hi, hF, hU, hW = host
    dr, dc, dw, di, dF, dU, dW = [x.cuda() for x in host]
    q, W0, kappa, dW0dR, dW0dG, dKdR, Beta = vv10_pointwise(
        hr[0, hi], hr[1:, hi], hw[hi], pars)
    xyz, gq, gw0, gk = _points(dr, dc, dw, di, pars)
    assert torch.equal(xyz.cpu(), hc[hi].to(torch.float32))
    for got, ref in ((gq, q), (gw0, W0), (gk, kappa)):
        assert got.dtype == torch.float32
        assert bool(((got.cpu().double() - ref).abs() <= 2.0 ** -23 * ref).all())
    exc = torch.ones(n, dtype=torch.float64, device='cuda')
    vv = torch.ones(4, ld, dtype=torch.float64, device='cuda')
    _add_potential(dr, di, pars, fac, dF, dU, dW, exc, vv)
    re, rv = torch.ones(n, dtype=torch.float64), torch.ones(4, ld, dtype=torch.float64)
    se, sv = re.clone(), rv.clone()
    re[hi] += fac * (Beta + 0.5 * hF)
    rv[0, hi] += 0.5 * fac * (Beta + hF + 1.5 * (hU * dKdR + hW * dW0dR))
    rv[1:, hi] += 3.0 * fac * hW * dW0dG * hr[1:, hi]
    # magnitudes: |dW0/dR| by its two terms, w2 = W0^2 - 4 pi / 3 R
    mag = (W0 ** 2 * 2.0 + 3.0 * np.pi * hr[0, hi]) / W0
    se[hi] += fac * (Beta + hF.abs())
    sv[0, hi] += fac * (Beta + hF.abs() + 1.5 * (hU.abs() * dKdR + hW.abs() * mag))
    sv[1:, hi] += (3.0 * fac * hW * dW0dG * hr[1:, hi]).abs()
    assert bool(((exc.cpu() - re).abs() <= 2.0 ** -46 * se).all())
    assert bool(((vv.cpu() - rv).abs() <= 2.0 ** -46 * sv).all())


@pytest.mark.gpu
@pytest.mark.parametrize('n', [1, 128, 1001])
def test_semilocal_kernel(n):
    import torch

    from pyscf_wb97mv_fast_gb300.scf import RshLdaVv10, _semilocal
    rng = np.random.default_rng(n)
    r = 10.0 ** rng.uniform(-16.0, 3.0, n)
    r[0] = 1e-14                                   # not above the threshold
    if n > 8:
        r[1:6] = [0.0, -1e-9, 5e-324, np.nan, 1.0000001e-14]
    f = RshLdaVv10(omega=0.3 if n < 500 else 0.6)
    host = torch.as_tensor(r)
    e, v = (x.cpu() for x in _semilocal(f, host.cuda()))
    re, rv = f.eval(host)
    live = host > 1e-14
    assert bool((e[~live] == 0).all()) and bool((v[~live] == 0).all())
    p = host[live]
    assert bool(((e - re)[live].abs() <= 2e-13 * p ** (4.0 / 3.0) + 1e-14 * p).all())
    assert bool(((v - rv)[live].abs() <= 2e-13 * p ** (1.0 / 3.0) + 1e-14).all())


def test_other_functionals_keep_their_eval():
    import torch

    from pyscf_wb97mv_fast_gb300.scf import RshLdaVv10, _semilocal

    class Mine(RshLdaVv10):
        def eval(self, rho):
            return rho, 2.0 * rho

    rho = torch.ones(3, dtype=torch.float64)
    assert torch.equal(_semilocal(Mine(), rho)[1], 2.0 * rho)
    f = RshLdaVv10()
    assert torch.equal(_semilocal(f, rho)[0], f.eval(rho)[0])
    f.eval = lambda r: (3.0 * r, r)
    assert torch.equal(_semilocal(f, rho)[0], 3.0 * rho)
