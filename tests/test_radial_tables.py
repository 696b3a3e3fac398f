'''The radial tables' arithmetic (lmb_radial.cuh) on the CPU against direct
sums in 64 bits: the pixels that are summed again in FP64.

Tolerance: 2e-5, the contract of the FP32 holograms, and the rounding of the
hologram itself to FP32.
'''
import numpy as np
import pytest

from oracle import field
from tests.cpu_harness.loader import Harness


@pytest.fixture(scope='module')
def h():
    return Harness()


def direct(h, c, p, a, n, kp, k):
    '''Field and hologram of one sphere at the pixels (2, npts) of z = 0.'''
    ab = h.sphere_ab(a, n, kp, 1.34, 0.447)
    E = h.field(np.vstack([c, np.zeros(c.shape[1])]), p, ab, k, fp64=True)
    return ab, E, np.sum(np.abs(E + np.array([[1], [0], [0]])) ** 2, axis=0)


def pixels(rng, n, far):
    '''Offsets from the axis, half of them within a tenth of far.'''
    r = np.concatenate([rng.uniform(0., .1 * far, n // 2),
                        rng.uniform(0., far, n - n // 2)])
    t = rng.uniform(0., 2. * np.pi, n)
    return np.stack([r * np.cos(t), r * np.sin(t)])


# behind large spheres of high index near the plane the field cancels
# between U and V rho^2 (the first four); and ordinary ones
SPHERES = [  # a_p, n_p, magnification, pixels from the sphere to the plane
    (6.30, 2.225, 0.048, 2.26), (20.5, 1.99, 0.048, 2.3),
    (19.7, 2.15, 0.03, 12.), (2.947, 2.109, 0.048, 2.61),
    (0.75, 1.45, 0.048, 2.1), (2.5, 1.8, 0.048, 40.)]


@pytest.mark.parametrize('a,n,mag,gap', SPHERES)
@pytest.mark.parametrize('side', [1., -1.])
def test_holograms_within_the_bound(h, a, n, mag, gap, side):
    k = field.wavenumber(1.34, 0.447, mag)
    c = pixels(np.random.default_rng(int(100 * a)), 6000, 60.)
    p = [0., 0., side * (a / mag + gap)]
    ab, _, H = direct(h, c, p, a, n, 0., k)
    _, got, _ = h.radial(c, p, ab, k)
    assert np.all(np.abs(got - H) <= 2e-5 + 6e-8 * H)
