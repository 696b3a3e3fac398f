'''GPU: calls whose radial tables find no memory take the direct sums, which
need none, instead of failing.'''
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def no_room(monkeypatch, times):
    '''The first allocations of bytes above 64 KB fail: the tables'
    scratch.'''
    import torch
    from pylorenzmie_b200.theory import _kernels as K
    refused = []

    class Torch:
        def __getattr__(self, name):
            return getattr(torch, name)

        @staticmethod
        def empty(*size, **kwargs):
            if kwargs.get('dtype') is torch.uint8 and size[0] > 1 << 16 \
                    and len(refused) < times:
                refused.append(size[0])
                raise torch.OutOfMemoryError('no room')
            return torch.empty(*size, **kwargs)
    monkeypatch.setattr(K, 'torch', Torch())
    return refused


@pytest.mark.parametrize('layered', [False, True])
@pytest.mark.parametrize('double', [False, True])
def test_images(layered, double, monkeypatch):
    from pylorenzmie_b200 import LayeredSphere, LorenzMie, Sphere
    s = LayeredSphere(a_p=1., n_p=1.5, fractions=(0.4,),
                      core_indices=(1.42,)) if layered else \
        Sphere(a_p=1., n_p=1.5)
    s.r_p = [500., 500., 200.]
    m = LorenzMie(coordinates=LorenzMie.meshgrid((1024, 1025)), particle=s,
                  double_precision=double)
    want = m.hologram()
    refused = no_room(monkeypatch, 1)
    got = m.hologram()
    assert refused
    assert np.abs(got - want).max() <= (1e-11 if double else 4e-5)


def test_gradient(monkeypatch):
    import torch
    from tests.test_gpu_vjp_small import inputs
    from pylorenzmie_b200.theory import autograd
    params, coords, g = inputs(401, 6, 1.5, False)
    h = autograd.hologram(params, coords)
    want, = torch.autograd.grad(h, params, g)
    refused = no_room(monkeypatch, 2)     # forward, backward
    h = autograd.hologram(params, coords)
    got, = torch.autograd.grad(h, params, g)
    assert len(refused) == 2
    _, J = autograd.jacobian(params.detach(), coords)
    scale = (J * g.double()[:, None]).abs().sum(-1)
    assert torch.all((got - want).abs() <= 1e-5 * scale)
