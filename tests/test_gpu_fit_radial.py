'''GPU: the fits' evaluation from radial tables (LMB_FIT_RADIAL) against the
evaluation that sums the orders at every pixel (launch shape 0).

Tolerances.  One evaluation at the start point gives chi^2 and, through
J^T J, the uncertainties: chi^2 within 1e-5, uncertainties within 1e-4 of
themselves.  Whole fits: both see the same data, and their holograms differ
by FP32 rounding, at most 2e-5 of noise 0.05, i.e. 4e-4 of a pixel's
standard deviation.  A shift common to all pixels moves a parameter by as
much of its uncertainty times the square root of the pixel count (100-300
here): bound 0.1 sigma.
'''
import numpy as np
import pytest

from pylorenzmie_b200 import _native

pytestmark = pytest.mark.gpu

FIVE = ('x_p', 'y_p', 'z_p', 'a_p', 'n_p')
SIX = FIVE + ('k_p',)


def fit(items, starts, config, variables=FIVE, layers=None, aberration=0.,
        reach=None, cap=None, evaluations=2000):
    from pylorenzmie_b200 import Instrument
    from pylorenzmie_b200.analysis import _fit
    inst = Instrument()
    packed = _fit.PackedFeatures(items)
    if reach is None:
        reach = int(np.ceil(packed.reach(starts)))
    cap = cap or _fit.fit_capacity(starts, inst.n_m, inst.wavelength, layers)
    f, d, c, p = _fit.upload(packed, starts)
    res, _ = _fit.fit_device(
        f, d, c, p, len(items), packed.total, inst, variables,
        dict(_fit.DEFAULT_SETTINGS, ftol=1e-8, xtol=1e-8,
             max_nfev=evaluations), cap, starts,
        tile_config=config, layers=layers, aberration=aberration, reach=reach)
    return (p.cpu().numpy().view(np.float64).reshape(-1, 6),
            res.cpu().numpy().view(_native.RESULT_DTYPE).copy())


def crops(shapes, z=200., seed=0, spherical=0., a=0.75):
    '''Items (data, grid, None) and starts, centred crops of one sphere.'''
    from pylorenzmie_b200 import AberratedLorenzMie, LorenzMie, workloads
    rng = np.random.default_rng(seed)
    items, starts = [], []
    for ny, nx in shapes:
        p = np.array([(nx - 1) / 2. + rng.uniform(-2, 2),
                      (ny - 1) / 2. + rng.uniform(-2, 2), z, a, 1.45, 1e-3])
        m = AberratedLorenzMie(coordinates=LorenzMie.meshgrid((ny, nx)),
                               spherical=spherical, double_precision=True)
        m.particle = workloads.spheres(p)[0]
        data = m.hologram() + rng.normal(0., 0.05, ny * nx)
        items.append((data.reshape(ny, nx), (0., 0., ny, nx), None))
        starts.append(p + [0.3, -0.2, 3., 0.01, 0.005, 0.])
    return items, np.array(starts)


def agree(items, starts, variables=FIVE, **kwargs):
    '''The tables' evaluation and fit against the direct sums'.'''
    idx = [SIX.index(v) for v in variables]
    options = {k: v for k, v in kwargs.items()
               if k in ('layers', 'aberration')}
    _, r = fit(items, starts, _native.LMB_FIT_RADIAL, variables,
               evaluations=1, **kwargs)
    _, s = fit(items, starts, 0, variables, evaluations=1, **options)
    np.testing.assert_allclose(r['dparams'][:, idx], s['dparams'][:, idx],
                               rtol=1e-4)
    np.testing.assert_allclose(r['redchi'], s['redchi'], rtol=1e-5)
    p, r = fit(items, starts, _native.LMB_FIT_RADIAL, variables, **kwargs)
    q, s = fit(items, starts, 0, variables, **options)
    assert np.all(r['status'] > 0) and np.all(s['status'] > 0)
    assert np.all(np.abs(p - q)[:, idx] <= 0.1 * s['dparams'][:, idx])


# edges of the 8x8 patches, of the bands of rows and of the part split
SHAPES = [(51, 51), (64, 64), (65, 63), (8, 300), (300, 8), (201, 201),
          (57, 129)]


@pytest.mark.parametrize('variables', [FIVE, SIX])
def test_grid_crops(variables):
    items, starts = crops(SHAPES)
    agree(items, starts, variables)


def test_pixel_lists_and_grids_together():
    items, starts = crops([(101, 101)] * 3, seed=1)
    rng = np.random.default_rng(3)
    for i, n in ((0, 900), (2, 4100)):
        keep = np.sort(rng.choice(101 * 101, n, replace=False))
        items[i] = (items[i][0].ravel()[keep], None,
                    np.stack([keep % 101, keep // 101]).astype(float))
    agree(items, starts)


def test_aberrated_below_the_plane_and_large():
    from pylorenzmie_b200 import Instrument
    inst = Instrument()
    c = 4. * inst.n_m ** 3 / inst.wavenumber() * 1.5
    items, starts = crops([(121, 121)] * 2, spherical=1.5, seed=2)
    agree(items, starts, aberration=c)
    items, starts = crops([(121, 121)], z=-180., seed=3)
    agree(items, starts)
    items, starts = crops([(301, 301)], z=300., a=2.5, seed=4)
    agree(items, starts)


def test_without_room_the_orders_are_summed_at_the_pixels():
    '''A reach too small for the tables, and a capacity of orders that
    leaves no room at all.'''
    items, starts = crops([(65, 65)], seed=5)
    agree(items, starts, reach=3)
    agree(items, starts, cap=1000)


def test_a_feature_does_not_depend_on_its_batch():
    '''One feature alone (many parts) and among others (few) to the bit.'''
    items, starts = crops([(121, 121)] * 40, seed=6)
    p, r = fit(items, starts, _native.LMB_FIT_RADIAL, reach=120)
    for i in (0, 17):
        q, s = fit(items[i:i + 1], starts[i:i + 1], _native.LMB_FIT_RADIAL,
                   reach=120)
        assert np.array_equal(p[i], q[0])
        assert np.array_equal(r['dparams'][i], s['dparams'][0])
