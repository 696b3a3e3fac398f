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


def nearest(a, n, kp, k, mag, fp64):
    '''The least distance of the plane from the sphere's centre (px) at
    which the library takes the tables.'''
    from pylorenzmie_b200 import _native
    lib = _native.load()
    flags = (_native.LMB_CARTESIAN | _native.LMB_BOHREN |
             (_native.LMB_FP64 if fp64 else 0))
    s = np.zeros(1, dtype=_native.SPHERE_DTYPE)

    def accepted(z):
        s[0] = 150., 150., z, a, n, kp
        return lib.lmb_radial_intervals(
            _native.Grid(0., 0., 0., 300, 300), 90000, s.ctypes.data, 1, k,
            mag, flags, 0.) > 0
    lo, hi = a / mag, a / mag + 100.
    assert accepted(hi) and not accepted(lo)
    while hi - lo > 1e-6:
        mid = 0.5 * (lo + hi)
        lo, hi = (lo, mid) if accepted(mid) else (mid, hi)
    return hi


@pytest.mark.parametrize('n,kp', [(1.36, 0.), (1.45, 0.), (2.6, 0.),
                                  (0.2, 3.)])
@pytest.mark.parametrize('fp64', [False, True])
def test_fields_wherever_the_tables_are_taken(h, n, kp, fp64):
    '''Within 1e-6 (FP64: 1e-12) of the field's largest component, the
    bounds of the fields of the library, as close to the plane as the library
    takes the tables, from spheres of a few nm on.'''
    k = field.wavenumber(1.34, 0.447, 0.048)
    rng = np.random.default_rng(7)
    for a in (0.005, 0.02, 0.05, 0.1, 0.2, 0.27, 0.3, 0.414, 0.5, 0.75, 2.5,
              6., 24.):
        c = pixels(rng, 400, 60.)
        p = [0., 0., nearest(a, n, kp, k, 0.048, fp64)]
        ab, E, _ = direct(h, c, p, a, n, kp, k)
        got, _, _ = h.radial(c, p, ab, k, fp64=fp64)
        err = np.abs(got - E).max() / np.abs(E).max()
        assert err <= (1e-12 if fp64 else 1e-6), (a, err)


@pytest.mark.parametrize('a,n,mag,gap', [
    (6.30, 2.225, 0.048, 2.26), (20.5, 1.99, 0.048, 2.3),
    (18.0170928, 2.33393022, 0.048, 50.3), (19.7, 2.15, 0.03, 12.)])
def test_pixels_summed_again_are_fp64(h, a, n, mag, gap):
    '''Half a unit in the last place of FP32, and 3e-9 of the hologram: the
    nodes are interpolated to 1e-9 of the field, and H is its square.'''
    k = field.wavenumber(1.34, 0.447, mag)
    c = pixels(np.random.default_rng(int(100 * a)), 6000, 30.)
    p = [0., 0., a / mag + gap]
    ab, _, H = direct(h, c, p, a, n, 0., k)
    _, got, marked = h.radial(c, p, ab, k)
    half = 0.5 * np.spacing(H.astype(np.float32)).astype(float)
    assert marked.any()
    assert np.all((np.abs(got - H) <= half + 3e-9 * H)[marked])
