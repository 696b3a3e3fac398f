'''GPU: gradients of few pixel-orders take the direct sums without asking for
the pixels' layout, those of many the tables; both against the Jacobian, the
holograms against FP64.

Tolerances: 2e-5, the contract of the FP32 holograms; 1e-5 of the largest term sum |g dH/dp| of a column, as between the
two ways: FP32 per pixel, Jacobians to ~3e-6 of the column maximum.
'''
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def inputs(side, n, a, listed, seed=0):
    import torch
    from pylorenzmie_b200 import LorenzMie
    rng = np.random.default_rng(seed)
    c = np.vstack([LorenzMie.meshgrid((side, side)),
                   np.zeros((1, side * side))])
    if listed:
        c = c[:, rng.random(side * side) < 0.67]
    p = np.zeros((n, 6))
    p[:, :2] = side / 2. + rng.uniform(-3., 3., (n, 2))
    p[:, 3], p[:, 4], p[:, 5] = a, 1.5, 1e-3
    p[:, 2] = a / 0.048 + rng.uniform(20., 300., n)
    g = rng.normal(size=(n, c.shape[1]))
    return (torch.from_numpy(p).cuda().requires_grad_(),
            torch.from_numpy(np.ascontiguousarray(c)).cuda(),
            torch.from_numpy(g).cuda().float())


@pytest.mark.parametrize('side,n,a,tables', [
    (51, 1, 0.5, False), (51, 12, 0.5, False), (201, 1, 0.9, False),
    (401, 1, 4., False),
    (401, 6, 1.5, True), (203, 12, 4., True)])   # 43 and 49 million
@pytest.mark.parametrize('listed', [False, True])
def test_gradient(side, n, a, tables, listed, monkeypatch):
    import torch
    from pylorenzmie_b200.theory import _kernels as K, autograd
    params, coords, g = inputs(side, n, a, listed)
    probes = []
    probe = K.probe_grid
    monkeypatch.setattr(K, 'probe_grid',
                        lambda c: probes.append(1) or probe(c))
    h = autograd.hologram(params, coords)
    got, = torch.autograd.grad(h, params, g)
    work = n * coords.shape[1] * K.nmax_cap_for(a, 1.5, 1e-3, 1.34, 0.447)
    assert bool(probes) == (work >= K.GRADIENT_TABLES)
    if not listed:
        assert bool(probes) == tables
    p = params.detach()
    _, J = autograd.jacobian(p, coords)
    d, inst, cap, ab, _, nmax = autograd._prepare(p, None)
    H = K.hologram(coords, d, torch.arange(n + 1, dtype=torch.int32).cuda(),
                   ab, nmax, cap, inst.wavenumber(), fp64=True)
    assert (h.detach().double() - H).abs().max() <= 2e-5
    terms = J * g.double()[:, None]
    scale = terms.abs().sum(-1)
    assert torch.all((got - terms.sum(-1)).abs() <= 1e-5 * scale)
