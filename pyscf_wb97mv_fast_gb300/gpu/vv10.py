"""VV10 non-local correlation on the GPU (reference:
pyscf_wb97mv_fast/gpu/vv10.py).

* ``Vv10Kernel.kernel_sum(coords, q, W0, kappa) -> (F, U, W)``: the
  O(N_g^2) double sum through the native tiled kernel (FP32 pair terms,
  Kahan inside a 256-point tile, FP64 across tiles, device-side tile-pair
  pruning when tile_tol > 0).  F is returned as -1.5 x the raw sum, the
  libdft VXC_vv10nlc convention the reference follows (:216-221).
* ``vv10_pointwise``: the per-point FP64 quantities of PySCF's _vv10nlc
  (reference :243-265) in torch; the flows below run them as one kernel
  before the double sum and one after it (wb_vv10_points,
  wb_vv10_potential).
* ``gpu_nr_nlc_vxc``: same signature and result as
  ``NumInt.nr_nlc_vxc`` -> (nelec, excsum, vmat) (reference :268-342): AO
  values and gradients (FP64, native), GGA density, threshold
  rho >= 1e-8, pointwise terms, kernel_sum, the GGA potential and the Fock
  contraction vmat = X^T (w v) X + transpose, all on the device in FP64
  except the pair sum.
"""
import math

import numpy as np

from pyscf_wb97mv_fast_gb300 import _native
from pyscf_wb97mv_fast_gb300.cosx import (CosxEngine, as_molecule, device_arg, device_out,
                                          round32)

THRESH = 1e-8
Unsupported = _native.Unsupported


def _torch():
    import torch
    return torch


class Vv10Kernel:
    """The double sum; tile_tol > 0 enables device-side tile-pair pruning."""

    def __init__(self, tile_tol=0.0):
        self.tile_tol = float(tile_tol)
        self.last_pairs_kept = None

    def kernel_sum(self, coords, q, W0, kappa):
        """coords (P, 3), q, W0, kappa (P,) on the device -> F, U, W FP64."""
        torch = _torch()
        _check_points(coords, 'coords')
        dev = coords.device
        n = int(coords.shape[0])
        F = torch.zeros(n, dtype=torch.float64, device=dev)
        U = torch.zeros_like(F)
        W = torch.zeros_like(F)
        if n == 0:
            self.last_pairs_kept = (0, 0)
            return F, U, W
        xyz = coords.to(torch.float32).contiguous()
        q32, w32, k32 = (_per_point(a, n, dev, name) for a, name in
                         ((q, 'q'), (W0, 'W0'), (kappa, 'kappa')))
        kept = _native.ctypes.c_int64()
        stream = _native.ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
        _native.check(_native.lib().wb_vv10_kernel_sum(
            _native.ptr(xyz), _native.ptr(q32), _native.ptr(w32), _native.ptr(k32),
            n, self.tile_tol, _native.ptr(F), _native.ptr(U), _native.ptr(W),
            stream, _native.ctypes.byref(kept)), 'wb_vv10_kernel_sum')
        self.last_pairs_kept = (int(kept.value), n * n)
        return F, U, W


    def kernel_sum_batch(self, coords, q, W0, kappa):
        """The double sums of several molecules in one launch: lists of
        per-molecule device arrays as kernel_sum takes them -> lists of F,
        U, W (each molecule's sums over its own points only; bitwise equal
        to kernel_sum per molecule)."""
        torch = _torch()
        if not coords or not len(coords) == len(q) == len(W0) == len(kappa):
            raise ValueError('one coords, q, W0 and kappa array per molecule')
        for c in coords:
            _check_points(c, 'coords')
        sizes = [int(c.shape[0]) for c in coords]
        dev = coords[0].device
        if any(c.device != dev for c in coords):
            raise ValueError('coords of one batch must share a device')
        offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        n = int(offsets[-1])
        xyz = torch.cat([c.to(torch.float32) for c in coords]).contiguous()
        q32, w32, k32 = (torch.cat([_per_point(a, m, dev, name)
                                    for a, m in zip(arrs, sizes)]).contiguous()
                         for arrs, name in ((q, 'q'), (W0, 'W0'), (kappa, 'kappa')))
        F = torch.zeros(n, dtype=torch.float64, device=dev)
        U = torch.zeros_like(F)
        W = torch.zeros_like(F)
        kept = _native.ctypes.c_int64()
        stream = _native.ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream)
        _native.check(_native.lib().wb_vv10_kernel_sum_batch(
            len(sizes), offsets.ctypes.data_as(_native.ctypes.c_void_p),
            _native.ptr(xyz), _native.ptr(q32), _native.ptr(w32), _native.ptr(k32),
            self.tile_tol, _native.ptr(F), _native.ptr(U), _native.ptr(W), stream,
            _native.ctypes.byref(kept)), 'wb_vv10_kernel_sum_batch')
        self.last_pairs_kept = (int(kept.value), int(sum(m * m for m in sizes)))
        sl = [slice(int(offsets[i]), int(offsets[i + 1])) for i in range(len(sizes))]
        return [F[x] for x in sl], [U[x] for x in sl], [W[x] for x in sl]


def _check_points(coords, name):
    """coords must be an (n, 3) torch tensor on a CUDA device: the kernels
    read its raw pointer."""
    torch = _torch()
    if not isinstance(coords, torch.Tensor) or not coords.is_cuda:
        raise ValueError('%s must be a torch tensor on a CUDA device' % name)
    if coords.dim() != 2 or coords.shape[1] != 3:
        raise ValueError('%s has shape %s, expected (n, 3)'
                         % (name, tuple(coords.shape)))


def _per_point(a, n, dev, name):
    """A per-point array (n,) as contiguous FP32 on dev."""
    torch = _torch()
    t = torch.as_tensor(a, device=dev).to(torch.float32).contiguous()
    if t.dim() != 1 or t.shape[0] != n:
        raise ValueError('%s has shape %s, expected (%d,)' % (name, tuple(t.shape), n))
    return t


def _constants(nlc_pars):
    """K, C and Beta of the parameters (b, C)."""
    Bvv, Cvv = nlc_pars
    pi = math.pi
    return (Bvv * 1.5 * pi * (9.0 * pi) ** (-1.0 / 6.0), Cvv,
            ((3.0 / (Bvv * Bvv)) ** 0.75) / 32.0)


def vv10_pointwise(rho0, grad, weights, nlc_pars):
    """Per-point FP64 terms on the thresholded set: q, W0, kappa, dW0/dR,
    dW0/dG, dK/dR, Beta (torch tensors; Beta a float)."""
    Kvv, Cvv, Beta = _constants(nlc_pars)
    pi43 = 4.0 * math.pi / 3.0
    R = rho0
    G = (grad ** 2).sum(dim=0)
    W0tmp = Cvv * (G / (R * R)) ** 2
    W0 = (W0tmp + pi43 * R).sqrt()
    dW0dR = (0.5 * pi43 * R - 2.0 * W0tmp) / W0
    dW0dG = W0tmp * R / (G * W0)
    kappa = Kvv * R ** (1.0 / 6.0)
    dKdR = kappa / 6.0
    q = R * weights
    return q, W0, kappa, dW0dR, dW0dG, dKdR, Beta


def _points(rho, coords, weights, ind, nlc_pars):
    """The double sum's inputs (xyz, q, W0, kappa) FP32 at the points ind
    (int64) of a grid: vv10_pointwise's quantities as one kernel
    (wb_vv10_points).  rho (4, ld), coords (n, 3), weights (n,) FP64."""
    torch = _torch()
    dev = rho.device
    nk, n = int(ind.shape[0]), int(weights.shape[0])
    kvv, cvv, _ = _constants(nlc_pars)
    rho = device_arg(rho, 'rho', torch.float64, dev, (4, None))
    coords = device_arg(coords, 'coords', torch.float64, dev, (n, 3))
    weights = device_arg(weights, 'weights', torch.float64, dev, (n,))
    ind = device_arg(ind, 'ind', torch.int64, dev, (nk,))
    out = [torch.empty((nk, 3) if i == 0 else nk, dtype=torch.float32, device=dev)
           for i in range(4)]
    _native.check(_native.lib().wb_vv10_points(
        _native.ptr(rho), int(rho.shape[1]), _native.ptr(coords), _native.ptr(weights),
        _native.ptr(ind), nk, kvv, cvv, *[_native.ptr(o) for o in out], CosxEngine._stream()), 'wb_vv10_points')
    return out


def _add_potential(rho, ind, nlc_pars, fac, F, U, W, exc, vv):
    """Adds fac times the energy density to exc (n,) and the derivatives to
    vv (4, ld) (half of d/d rho, and d/d grad) from the double sums at the
    points ind (wb_vv10_potential)."""
    torch = _torch()
    dev = rho.device
    nk = int(ind.shape[0])
    kvv, cvv, beta = _constants(nlc_pars)
    F, U, W = (device_arg(x.to(torch.float64), 'sum', torch.float64, dev, (nk,))
               for x in (F, U, W))
    rho = device_arg(rho, 'rho', torch.float64, dev, (4, None))
    device_out(vv, 'vv', torch.float64, dev, tuple(rho.shape))
    device_out(exc, 'exc', torch.float64, dev, tuple(exc.shape))
    _native.check(_native.lib().wb_vv10_potential(
        _native.ptr(rho), int(rho.shape[1]), _native.ptr(ind), nk, kvv, cvv,
        beta, float(fac), _native.ptr(F), _native.ptr(U), _native.ptr(W),
        _native.ptr(exc), _native.ptr(vv), CosxEngine._stream()), 'wb_vv10_potential')


def _sum_inputs(kernel, rho, coords, weights, ind, nlc_pars):
    """What kernel.kernel_sum is given at the points ind: FP32 from one kernel
    (_points) for Vv10Kernel's own sum, which works on those; for a caller's
    kernel the coordinates in FP32 and q, W0 and kappa in FP64."""
    torch = _torch()
    if getattr(kernel.kernel_sum, '__func__', None) is Vv10Kernel.kernel_sum:
        return _points(rho, coords, weights, ind, nlc_pars)
    q, W0, kappa = vv10_pointwise(rho[0, ind], rho[1:4, ind], weights[ind], nlc_pars)[:3]
    return coords[ind].to(torch.float32), q, W0, kappa


class Vv10Context:
    """Per-mf state of the VV10 flow: the native engine (AO tables) and the
    kernel-sum settings."""

    def __init__(self, mol, tile_tol=0.0, device=None):
        self.mol = mol
        self.tile_tol = float(tile_tol)
        self.device = device
        self.engine = None
        self.kernel = Vv10Kernel(tile_tol)

    def build(self):
        if self.engine is None:
            self.engine = CosxEngine(as_molecule(self.mol), device=self.device)
        return self.engine


def _prepare_dm(dm, hermi):
    dm = np.asarray(dm, dtype=np.float64)
    if dm.ndim == 3 and dm.shape[0] == 1:
        dm = dm[0]
    if dm.ndim != 2 or dm.shape[0] != dm.shape[1]:
        raise Unsupported(_native.WB_ERR_UNSUPPORTED,
                          'GPU VV10 supports a single RKS density matrix')
    if hermi != 1:
        dm = 0.5 * (dm + dm.T)
    return dm


def vv10_prepare(eng, g, D, nlc_pars, gemm='fp64', kernel=None):
    """The steps of vv10_energy_fock before the double sum (the GGA density
    on the NLC grid g, the threshold and the pointwise terms): a state for
    vv10_finish; st['xyz'], st['q'], st['W0'], st['kappa'] are the double
    sum's inputs (Vv10Kernel.kernel_sum or, for several molecules,
    kernel_sum_batch; or kernel's kernel_sum, see _sum_inputs).  gemm as in
    vv10_energy_fock."""
    torch = _torch()
    if gemm not in ('fp64', 'split64', 'fp32'):
        raise ValueError("gemm must be 'fp64', 'split64' or 'fp32'")
    n = g.n
    w = g.weights
    X = g.X
    if gemm == 'fp32':
        T = eng.ozaki_f(X[0], D)
    elif gemm == 'split64':
        T = eng.ozaki_f(X[0], D, fp64=True)
    else:
        if int(X.shape[2]) != round32(n):       # a grid padded to another length
            X = torch.nn.functional.pad(X[:, :, :n], (0, round32(n) - n))
        T = eng.gemm64_f(X[0], D.T)
    rho = eng.gga_rho(X, T, n)                            # (4, ld)
    ind = torch.nonzero(rho[0, :n] >= THRESH).squeeze(1)
    xyz, q, W0, kappa = _sum_inputs(kernel or Vv10Kernel(0.0), rho, g.coords, w, ind,
                                    nlc_pars)
    return dict(eng=eng, g=g, X=X, gemm=gemm, n=n, rho=rho, ind=ind, nlc_pars=nlc_pars,
                xyz=xyz, q=q, W0=W0, kappa=kappa)


def vv10_finish(st, F, U, W):
    """E_nl and V_nl from a vv10_prepare state and the double sums F, U, W
    of its points."""
    torch = _torch()
    eng, X, n, ind, rho = (st[k] for k in ('eng', 'X', 'n', 'ind', 'rho'))
    w = st['g'].weights
    exc = torch.zeros(n, dtype=torch.float64, device=rho.device)
    vv = torch.zeros_like(rho)
    _add_potential(rho, ind, st['nlc_pars'], 1.0, F, U, W, exc, vv)
    e_nl = (rho[0, :n] * w * exc).sum()
    # G = 1/2 v0 X0 + sum_d 2 v1 grad_d X_d, then X0^T (w o G); G FP64, or
    # rounded once to FP32 (gemm 'fp32')
    G = eng.gga_aow(X, vv, n, torch.float32 if st['gemm'] == 'fp32' else None)
    if st['gemm'] == 'fp64':
        vmat = eng.gemm64_k(X[0], G, w)
    else:
        vmat = eng.ozaki_k(X[0], G, w)
    return e_nl, vmat + vmat.T


def vv10_energy_fock(eng, g, D, nlc_pars, kernel=None, fp32=False, gemm='fp64'):
    """E_nl and V_nl of one density on a device grid, all on the device:
    g holds coordinates (engine frame), weights and the deriv-1 AO values
    X (4, nao, ld) (scf.DeviceGrid); D (nao, nao) FP64 device.  The same
    steps as gpu_nr_nlc_vxc for one parameter set (b, C) with factor 1:
    GGA density, threshold rho >= 1e-8, pointwise terms, the pair sum, the
    GGA potential and vmat = X^T (w v) X + transpose.  Returns (E_nl
    device scalar, V_nl (nao, nao)).  The two GEMMs (D X and the Fock
    side) run as gemm:
      'fp64'    FP64 GEMMs (CosxEngine.gemm64_f / gemm64_k);
      'split64' the bf16 Ozaki split with FP64 operands and results (42
                bits of the per-row / per-column maxima), the SCF's FP64
                tail;
      'fp32'    the split with D X rounded once to FP32 and the Fock side
                from an FP32-rounded G, the SCF's FP32 stages (fp32=True
                is the same)."""
    kernel = kernel or Vv10Kernel(0.0)
    st = vv10_prepare(eng, g, D, nlc_pars, 'fp32' if fp32 else gemm, kernel)
    F, U, W = kernel.kernel_sum(st['xyz'], st['q'], st['W0'], st['kappa'])
    return vv10_finish(st, F, U, W)


def gpu_nr_nlc_vxc(ctx, ni, mol, grids, xc_code, dm, relativity=0, hermi=1,
                   max_memory=2000, verbose=None):
    """GPU replacement of NumInt.nr_nlc_vxc (RKS ground state)."""
    torch = _torch()
    if relativity not in (0, None):
        raise Unsupported(_native.WB_ERR_UNSUPPORTED,
                          'relativistic NLC not supported')
    dm = _prepare_dm(dm, hermi)
    nlc_coefs = ni.nlc_coeff(xc_code)
    if not nlc_coefs:
        raise Unsupported(_native.WB_ERR_UNSUPPORTED,
                          '%r has no NLC parameter set' % (xc_code,))
    eng = ctx.build()
    dev = eng.device
    nao = eng.nao
    coords = eng.relative(np.asarray(grids.coords, dtype=np.float64))
    w = torch.as_tensor(np.asarray(grids.weights, dtype=np.float64), device=dev)
    n = int(coords.shape[0])
    X = eng.ao_eval_deriv1(coords)                        # (4, nao, ld)
    D = torch.as_tensor(dm, device=dev)
    rho = eng.gga_rho(X, eng.gemm64_f(X[0], D.T), n)      # (4, ld)
    rho0 = rho[0, :n]
    exc = torch.zeros(n, dtype=torch.float64, device=dev)
    vv = torch.zeros_like(rho)          # d/d rho (half of it) and d/d grad
    ind = torch.nonzero(rho0 >= THRESH).squeeze(1)
    for nlc_pars, fac in nlc_coefs:
        F, U, W = ctx.kernel.kernel_sum(
            *_sum_inputs(ctx.kernel, rho, coords, w, ind, nlc_pars))
        _add_potential(rho, ind, nlc_pars, fac, F, U, W, exc, vv)
    # vmat = X0^T (w o G) + its transpose, G = 1/2 v0 X0 + sum_d v_d X_d
    vmat = eng.gemm64_k(X[0], eng.gga_aow(X, vv, n), w)
    vmat = vmat + vmat.T
    nelec = float((rho0 * w).sum())
    excsum = float((rho0 * w * exc).sum())
    return nelec, excsum, vmat.cpu().numpy()
