'''GPU: holograms behind large spheres of high index near the plane, where
the field cancels between U and V rho^2 (lmb_radial.cuh), as grids and as
pixel lists, against FP64.

Tolerance: 2e-5, the contract of the FP32 holograms, and the rounding of the
hologram itself to FP32.
'''
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPHERES = [  # a_p, n_p, magnification, pixels from the sphere to the plane
    (6.30, 2.225, 0.048, 2.26), (20.5, 1.99, 0.048, 2.3),
    (19.7, 2.15, 0.03, 12.)]


@pytest.mark.parametrize('listed', [False, True])
@pytest.mark.parametrize('a,n,mag,gap', SPHERES)
def test_bright_pixels_match_fp64(a, n, mag, gap, listed):
    from pylorenzmie_b200 import Instrument, LorenzMie, Sphere
    c = LorenzMie.meshgrid((200, 203))
    if listed:
        c = c[:, ::2] + 0.25
    s = Sphere(a_p=a, n_p=n)
    s.r_p = [100.3, 99.6, a / mag + gap]
    inst = Instrument(magnification=mag)
    h32, h64 = (LorenzMie(coordinates=c, particle=s, instrument=inst,
                          double_precision=d).hologram()
                for d in (False, True))
    assert np.all(np.abs(h32 - h64) <= 2e-5 + 6e-8 * h64)


@pytest.mark.parametrize('double', [False, True])
@pytest.mark.parametrize('a,n,z', [
    (0.02, 1.45, 2.5), (0.1, 1.45, 4.2), (0.3, 2.6, 8.3),   # summed directly
    (0.02, 1.45, 14.5), (0.3, 2.6, 14.5), (0.75, 1.45, 22.)])   # tables
def test_small_spheres_near_the_plane(a, n, z, double):
    '''Fields within 1e-6 (FP64: 1e-12) of the largest component of the
    direct FP64 sums.'''
    from pylorenzmie_b200 import LorenzMie, Sphere
    c = LorenzMie.meshgrid((200, 203))
    s = Sphere(a_p=a, n_p=n)
    s.r_p = [100.3, 99.6, z]
    ref = LorenzMie(coordinates=c, particle=s, double_precision=True)
    ref._coords
    ref._grid_dev = (None,)                     # direct sums
    E = ref.field()
    got = LorenzMie(coordinates=c, particle=s, double_precision=double).field()
    err = np.abs(got - E).max() / np.abs(E).max()
    assert err <= (1e-12 if double else 1e-6)
