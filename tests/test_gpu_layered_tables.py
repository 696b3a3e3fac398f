'''GPU: images of layered spheres take the radial tables from IMAGE_TABLES
pixel-orders on, direct sums below; both against FP64 (2e-5, the contract of
the FP32 holograms).
'''
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('shape,n,tables', [
    ((64, 64), 1, False), ((301, 300), 1, False), ((257, 255), 4, False),
    ((640, 641), 3, True), ((1024, 1025), 2, True)])
def test_layered_images(shape, n, tables, monkeypatch):
    from pylorenzmie_b200 import LayeredSphere, LorenzMie, _native
    ny, nx = shape
    rng = np.random.default_rng(n)
    spheres = []
    for _ in range(n):
        s = LayeredSphere(a_p=rng.uniform(0.8, 1.2), n_p=1.5,
                          fractions=(0.4,), core_indices=(1.42,))
        s.r_p = [rng.uniform(0., nx), rng.uniform(0., ny),
                 rng.uniform(100., 300.)]
        spheres.append(s)
    c = LorenzMie.meshgrid(shape)
    calls = []
    lib = _native.load()
    grid = lib.lmb_hologram_grid
    monkeypatch.setattr(lib, 'lmb_hologram_grid',
                        lambda *a: calls.append(1) or grid(*a))
    h32 = LorenzMie(coordinates=c, particle=spheres).hologram()
    assert bool(calls) == tables
    ref = LorenzMie(coordinates=c, particle=spheres, double_precision=True)
    ref._coords
    ref._grid_dev = (None,)                     # direct sums
    assert np.abs(h32 - ref.hologram()).max() <= 2e-5
