'''Differentiable holograms: torch.autograd.Function over the CUDA kernels.

``hologram(params, coordinates, instrument)`` returns the (B, npts) FP32
holograms of B single spheres, params (B, 6) = (x_p, y_p, z_p, a_p, n_p,
k_p).  Its backward pass is a hand-written VJP kernel that reduces
g * dH/dparam over the pixels, from radial tables of the hologram's
derivatives where the pixels lie in a plane clear of the spheres
(``lmb_hologram_vjp_grid``), else from recurrences run again pixel by pixel
(``lmb_hologram_vjp``).  Nothing per order or per pixel is stored between
forward and backward (only the O(n_max) Mie coefficients and their parameter
derivatives).
``jacobian`` returns the full per-pixel 6-column Jacobian instead.

No reference counterpart runs here: the reference torch backend is not
differentiable (theory/torchLorenzMie.py:293-300); its JAX backend's
jacfwd (theory/jaxLorenzMie.py:283-286) is the analogue.
'''
import numpy as np
import torch

from . import _kernels as K
from .Instrument import Instrument


def _prepare(params, instrument, host=None):
    p = params.detach().to(torch.float64).contiguous()
    inst = instrument or Instrument()
    if host is None:
        host = p.cpu().numpy()
    cap = K.nmax_cap_for(host[:, 3], host[:, 4], host[:, 5], inst.n_m,
                         inst.wavelength)
    # the capacity covers these spheres, so the coefficients can fail only on
    # invalid parameters: checked here, without reading the device again
    if not (np.isfinite(host).all() and (host[:, 3] > 0.).all()):
        raise ValueError('sphere parameters must be finite with a_p > 0')
    ab, dab, nmax = K.sphere_ab(p, inst.n_m, inst.wavelength, cap, deriv=True,
                                check=False)
    return p, inst, cap, ab, dab, nmax


def _coords(coordinates, device):
    c = torch.as_tensor(coordinates, dtype=torch.float64, device=device)
    if c.shape[0] == 2:
        c = torch.cat([c, torch.zeros((1, c.shape[1]), dtype=torch.float64,
                                      device=device)])
    return c.contiguous()


class HologramFunction(torch.autograd.Function):
    '''H(params) with dH/dparams from the VJP kernel.'''

    @staticmethod
    def forward(ctx, params, coordinates, instrument, bohren):
        # the parameters and the pixels' layout in one read-back
        B, npts = params.shape[0], coordinates.shape[1]
        grid, host = None, None
        if B and npts:
            both = torch.cat([
                params.detach().to(torch.float64).reshape(-1),
                coordinates[2, :1],
                K.probe_grid(coordinates).view(torch.float64)]).cpu().numpy()
            host = both[:6 * B].reshape(B, 6).copy()
            grid = K.make_grid(both[6 * B], npts,
                               both[6 * B + 1:].view(np.int64))
        p, inst, cap, ab, dab, nmax = _prepare(params, instrument, host)
        item_start = torch.arange(B + 1, dtype=torch.int32, device=p.device)
        h = None
        records = None if grid is None else host.view(K.SPHERE_DTYPE).ravel()
        if grid is not None:
            h = K.on_grid(grid, coordinates, records, p, item_start, ab, nmax,
                          cap, inst, True, bohren, 0.)
        if h is None:
            h = K.hologram(coordinates, p, item_start, ab, nmax, cap,
                           inst.wavenumber(), True, bohren, False)
        ctx.save_for_backward(p, coordinates, ab, dab, nmax)
        ctx.inst, ctx.cap, ctx.bohren = inst, cap, bohren
        ctx.grid, ctx.records = grid, records
        return h

    @staticmethod
    def backward(ctx, gout):
        p, coordinates, ab, dab, nmax = ctx.saved_tensors
        grad = None
        if ctx.grid is not None:
            grad = K.vjp_on_grid(ctx.grid, coordinates, ctx.records, p, ab,
                                 dab, nmax, ctx.cap, ctx.inst, gout,
                                 ctx.bohren)
        if grad is None:
            grad = K.hologram_vjp(coordinates, p, ab, dab, nmax, ctx.cap,
                                  ctx.inst.wavenumber(), gout.contiguous(),
                                  ctx.bohren)
        return grad.to(p.dtype), None, None, None


def hologram(params, coordinates, instrument=None, bohren=True):
    '''Differentiable (B, npts) float32 holograms of B spheres.'''
    if params.dim() == 1:
        params = params.unsqueeze(0)
    c = _coords(coordinates, params.device)
    return HologramFunction.apply(params, c, instrument, bohren)


def jacobian(params, coordinates, instrument=None, bohren=True):
    '''Holograms (B, npts) and Jacobians (B, 6, npts), float64 tensors.'''
    if params.dim() == 1:
        params = params.unsqueeze(0)
    p, inst, cap, ab, dab, nmax = _prepare(params, instrument)
    c = _coords(coordinates, p.device)
    return K.jacobian(c, p, ab, dab, nmax, cap, inst.wavenumber(), bohren)
