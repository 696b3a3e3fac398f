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
