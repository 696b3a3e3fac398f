'''GPU: gradients of holograms from radial tables (lmb_hologram_vjp_grid)
against the VJP kernel that sums the orders at every pixel.

Tolerance: 1e-5 of the largest term sum |g dH/dp| of a column: both sums
are FP32 per pixel, with Jacobians to ~3e-6 of the column maximum.
'''
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape,z0,a,bohren', [
    ((64, 64), 0., 0.75, True), ((65, 203), 0., 1.2, True),
    ((201, 201), 5., 0.9, True), ((129, 97), 0., 0.6, False),
    ((401, 401), 0., 5., True), ((9, 700), 0., 0.8, True)])
@pytest.mark.parametrize('listed', [False, True])
def test_gradient_matches_direct_sums(shape, z0, a, bohren, listed):
    import torch
    from pylorenzmie_b200 import Instrument, LorenzMie
    from pylorenzmie_b200.theory import _kernels as K, autograd
    ny, nx = shape
    rng = np.random.default_rng(ny)
    c = np.vstack([LorenzMie.meshgrid(shape), np.full((1, ny * nx), z0)])
    if listed:                   # two thirds of the pixels: not a grid
        c = c[:, rng.random(ny * nx) < 0.67]
    p = np.zeros((3, 6))
    p[:, 0] = nx / 2. + rng.uniform(-3., 3., 3)
    p[:, 1] = ny / 2. + rng.uniform(-3., 3., 3)
    p[:, 2] = a / 0.048 + z0 + np.array([20., 120., 300.])
    p[:, 3], p[:, 4], p[:, 5] = a, 1.5, 1e-3
    coords = torch.from_numpy(np.ascontiguousarray(c)).cuda()
    params = torch.from_numpy(p).cuda().requires_grad_()
    g = torch.from_numpy(rng.normal(size=(3, c.shape[1]))).cuda().float()
    h = autograd.hologram(params, coords, bohren=bohren)
    got, = torch.autograd.grad(h, params, g)
    d, inst, cap, ab, dab, nmax = autograd._prepare(params, None)
    ref = K.hologram_vjp(coords, d, ab, dab, nmax, cap, inst.wavenumber(), g,
                         bohren)
    _, J = K.jacobian(coords, d, ab, dab, nmax, cap, inst.wavenumber(), bohren)
    scale = (J * g.double()[:, None]).abs().sum(-1)
    assert torch.all((got - ref).abs() <= 1e-5 * scale)
    # and the tables were used
    grid = K.make_grid(z0, c.shape[1], K.probe_grid(coords).cpu().numpy())
    records = p.view(K.SPHERE_DTYPE).ravel()
    tab = K.vjp_on_grid(grid, coords, records, d, ab, dab, nmax, cap, inst, g,
                        bohren)
    assert tab is not None and torch.equal(tab, got)
