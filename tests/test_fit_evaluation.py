'''Which evaluation a batch of fits takes (no GPU): radial tables with room for
the fastest hologram of the batch, launch shapes where a quarter of the
spheres or more are too near the plane, or the crops too large.'''
import numpy as np
import pytest

from pylorenzmie_b200 import Instrument, _native
from pylorenzmie_b200.analysis import _fit

K = Instrument().wavenumber()


def starts(n, z=200., a=0.75):
    p = np.zeros((n, 6))
    p[:] = (100., 100., z, a, 1.45, 0.)
    return p


def reach(p, far=150., aberration=0.):
    return _native.load().lmb_fit_radial_reach(
        p.ctypes.data, len(p), far, K, 0.048, aberration)


def evaluation(p, side):
    packed = _fit.PackedFeatures(
        [(np.zeros((side, side), np.float32), (0., 0., side, side), None)] *
        len(p))
    cap = _fit.fit_capacity(p, 1.34, 0.447)
    return _fit.evaluation(packed, p, Instrument(), ('z_p',), cap, None, None,
                           False, 0.)


def test_reach():
    r = reach(starts(3))
    assert 150 <= r <= 151
    assert reach(starts(3, z=-200.)) == r
    # the plane 3 px from a sphere of 21 px: oscillations above k
    assert 1.3 * 150 < reach(starts(3, z=24., a=1.)) < 1.7 * 150
    assert reach(starts(3), aberration=500.) > r
    for bad in (starts(3, z=12., a=0.3), starts(3, z=5.), starts(3, z=np.nan),
                starts(3, a=-1e9)):
        assert reach(bad) in (0, r)
    assert reach(starts(3, z=12., a=0.3)) == 0
    assert reach(starts(3, z=np.nan)) == 0
    assert reach(starts(3), far=450.) == 0
    assert reach(starts(3), far=np.inf) == 0 and reach(starts(3), far=np.nan) == 0


@pytest.mark.parametrize('n,near,tables', [(1, 1, False), (8, 1, True),
                                           (8, 2, False), (256, 63, True),
                                           (256, 64, False)])
def test_some_spheres_near_the_plane(n, near, tables):
    p = starts(n)
    p[:near, 2:4] = 12., 0.3
    assert (reach(p) > 0) == tables


@pytest.mark.parametrize('n,side,z,a,radial', [
    (1, 201, 200., 0.75, True), (1, 51, 200., 0.75, False),
    (64, 51, 200., 0.75, True), (1, 201, 12., 0.3, False),
    (256, 201, 24., 1., True), (64, 801, 200., 0.75, False)])
def test_evaluation(n, side, z, a, radial):
    p = starts(n, z, a)
    p[:, :2] = side / 2.
    config, room = evaluation(p, side)
    assert (config == _native.LMB_FIT_RADIAL) == radial
    assert (room > 0) == radial
    if not radial:
        assert config == _fit.default_shape(n)
