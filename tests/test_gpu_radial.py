'''GPU: fields and holograms on pixel grids from radial tables
(lmb_hologram_grid, lmb_field_grid) against the direct FP64 sums, and which
images take that path.

Tolerances.  Holograms: 2e-5 absolute, the contract of the FP32 holograms.
Fields: 1e-6 of the sum of the particles' largest components.  The table is
off by at most 4e-8 of a component (FP64 nodes, degree-5 polynomials) and
its FP32 evaluation by a few roundings of 6e-8.
'''
import numpy as np
import pytest


def grid_model(shape, particles, **kwargs):
    from pylorenzmie_b200 import LorenzMie, AberratedLorenzMie
    cls = AberratedLorenzMie if 'spherical' in kwargs else LorenzMie
    return cls(coordinates=LorenzMie.meshgrid(shape), particle=particles,
               **kwargs)


def uses_tables(model, spheres, bohren):
    '''Whether lmb_render_plan chooses the tables for these images.'''
    from pylorenzmie_b200 import _native
    from pylorenzmie_b200.theory import _kernels as K
    from pylorenzmie_b200.theory.LorenzMie import _records
    rec = _records(spheres)
    inst = model.instrument
    plan = _native.Render()
    grid, full = model._grid
    assert full and _native.load().lmb_render_plan(
        grid, 0, model.coordinates.shape[1], rec.ctypes.data, len(rec), 1,
        inst.n_m, inst.wavelength, inst.wavenumber(), inst.magnification,
        K._flags(True, bohren, model.double_precision), model._aberration(),
        plan) == _native.LMB_OK
    return plan.intervals > 0


def rows(n, shape, seed, below=False):
    rng = np.random.default_rng(seed)
    p = np.zeros((n, 6))
    p[:, 0] = rng.uniform(-20., shape[1] + 20., n)
    p[:, 1] = rng.uniform(-20., shape[0] + 20., n)
    p[:, 3] = rng.uniform(0.3, 2.5, n)
    p[:, 4] = rng.uniform(1.36, 1.8, n)
    p[:, 5] = rng.uniform(0., 1e-2, n)
    # from 2 px above the sphere on, on either side of the focal plane
    p[:, 2] = p[:, 3] / 0.048 + 2. + rng.exponential(100., n)
    if below:
        p[::2, 2] *= -1.
    return p


CASES = [
    # shape, spheres, instrument, other options
    ((256, 256), 1, {}, {}),
    ((257, 255), 3, {}, {}),           # ragged tiles on both edges
    ((223, 289), 33, {}, {}),          # more than one group of particles
    ((225, 287), 4, {}, {'below': True}),
    ((256, 320), 2, {}, {'bohren': False}),
    ((256, 260), 2, {}, {'spherical': 1.5}),
    ((256, 260), 2, {'magnification': 0.135}, {}),   # few px an interval
    ((256, 260), 2, {'magnification': 0.02}, {}),
]


@pytest.mark.gpu
@pytest.mark.parametrize('shape,n,inst,opt', CASES)
def test_grid_images_match_fp64(shape, n, inst, opt):
    from pylorenzmie_b200 import Instrument, workloads
    opt = dict(opt)
    p = rows(n, shape, seed=n + len(opt), below=opt.pop('below', False))
    instrument = Instrument(**inst)
    if inst:
        p[:, 2] = np.sign(p[:, 2]) * (p[:, 3] / instrument.magnification +
                                      4. / instrument.wavenumber() + 30.)
    bohren = opt.pop('bohren', True)
    spheres = workloads.spheres(p)
    m32 = grid_model(shape, spheres, instrument=instrument, **opt)
    m64 = grid_model(shape, spheres, instrument=instrument,
                     double_precision=True, **opt)
    m64._coords
    m64._grid_dev = (None,)                     # direct sums
    h32 = m32.hologram(bohren=bohren)
    h64 = m64.hologram(bohren=bohren)
    assert uses_tables(m32, spheres, bohren)
    assert np.abs(h32 - h64).max() <= 2e-5
    f32, f64 = m32.field(bohren=bohren), m64.field(bohren=bohren)
    scale = sum(np.abs(m64.scattered_field(s, bohren=bohren)).max()
                for s in spheres)
    assert np.abs(f32 - f64).max() <= 1e-6 * scale


@pytest.mark.gpu
@pytest.mark.parametrize('shape,n,inst,opt', CASES)
def test_fp64_grid_images_match_direct_sums(shape, n, inst, opt):
    '''FP64 tables: 1e-12 of the sum of the particles' largest components
    (interpolation 1e-14, and the rounding of phases of ~10^3 rad at the
    nodes and at the pixels, ~1e-13 each).'''
    from pylorenzmie_b200 import Instrument, workloads
    opt = dict(opt)
    p = rows(n, shape, seed=n + len(opt), below=opt.pop('below', False))
    instrument = Instrument(**inst)
    if inst:
        p[:, 2] = np.sign(p[:, 2]) * (p[:, 3] / instrument.magnification +
                                      4. / instrument.wavenumber() + 30.)
    bohren = opt.pop('bohren', True)
    spheres = workloads.spheres(p)
    m = grid_model(shape, spheres, instrument=instrument,
                   double_precision=True, **opt)
    d = grid_model(shape, spheres, instrument=instrument,
                   double_precision=True, **opt)
    d._coords
    d._grid_dev = (None,)                       # direct sums
    f, ref = m.field(bohren=bohren), d.field(bohren=bohren)
    assert uses_tables(m, spheres, bohren)
    scale = sum(np.abs(d.scattered_field(s, bohren=bohren)).max()
                for s in spheres)
    assert np.abs(f - ref).max() <= 1e-12 * scale
    h, ref = m.hologram(bohren=bohren), d.hologram(bohren=bohren)
    assert np.abs(h - ref).max() <= 2e-12 * scale * (1. + scale)


@pytest.mark.gpu
def test_grid_batch_items():
    '''Items of different lengths, an empty one among them.'''
    from pylorenzmie_b200 import workloads
    shape = (256, 300)
    lists = [workloads.spheres(rows(n, shape, seed=n)) if n else []
             for n in (2, 0, 5, 1)]
    h32 = grid_model(shape, lists[0]).batch_hologram(lists)
    h64 = grid_model(shape, lists[0],
                     double_precision=True).batch_hologram(lists)
    assert np.abs(h32 - h64).max() <= 2e-5
    assert np.all(h32[1] == 1.) and np.all(h64[1] == 1.)


@pytest.mark.gpu
def test_grid_probe():
    import torch
    from pylorenzmie_b200 import LorenzMie
    from pylorenzmie_b200.theory import _kernels as K
    c = np.vstack([LorenzMie.meshgrid((40, 53), corner=(2.5, -7.)),
                   np.full((1, 40 * 53), 3.)])

    def probe(a):
        a = np.ascontiguousarray(a)
        found = K.probe_grid(torch.from_numpy(a).cuda()).cpu().numpy()
        host = K.probe_host(a)
        assert found[1] == 0 or host[1] > 0
        assert (found[2] > 0) == (host[2] > 0)
        if not found[2]:
            assert np.array_equal(found, host)
        return K.make_grid(a[2, 0], a.shape[1], found)
    g, full = probe(c)
    assert full and (g.x0, g.y0, g.z, g.nx, g.ny) == (2.5, -7., 3., 53, 40)
    for j, i, v in ((0, 700, 1e-12), (1, 2119, 1.)):
        bad = c.copy()
        bad[j, i] += v
        g, full = probe(bad)                    # a list in the plane
        assert not full and g.x0 == 2.5 and g.y0 == -7.
        assert g.x0 + g.nx - 1 >= bad[0].max()
        assert g.y0 + g.ny - 1 >= bad[1].max()
    assert not probe(c[:, :-1])[1]              # a ragged last row
    assert not probe(c[:, ::2])[1]              # every other pixel
    g, full = probe(c[:, :53])
    assert full and g.ny == 1
    for j, v in ((2, 1e-9), (0, np.nan), (1, np.inf)):
        bad = c.copy()
        bad[j, 5] += v
        assert probe(bad) is None               # not in one plane


@pytest.mark.gpu
@pytest.mark.parametrize('step', [2, 3])
def test_pixel_lists_match_fp64(step):
    '''Pixels of one plane that are not a grid, with fractions.'''
    from pylorenzmie_b200 import LorenzMie, workloads
    c = LorenzMie.meshgrid((480, 501))[:, ::step] + 0.25
    c[0, ::7] += 0.5
    spheres = workloads.spheres(rows(3, (480, 501), seed=step))
    m32 = LorenzMie(coordinates=c, particle=spheres)
    m64 = LorenzMie(coordinates=c, particle=spheres, double_precision=True)
    assert np.abs(m32.hologram() - m64.hologram()).max() <= 2e-5
    f32, f64 = m32.field(), m64.field()
    scale = sum(np.abs(m64.scattered_field(s)).max() for s in spheres)
    assert np.abs(f32 - f64).max() <= 1e-6 * scale


def test_rule_on_the_host():
    '''Where the tables do not apply the rule says so (no GPU needed).'''
    from pylorenzmie_b200 import _native
    lib = _native.load()
    k = 0.904
    cart = _native.LMB_CARTESIAN | _native.LMB_BOHREN

    def intervals(z_p=200., a_p=0.75, nx=300, ny=300, x0=0., flags=cart,
                  aberration=0., k=k, x_p=150.):
        s = np.zeros(1, dtype=_native.SPHERE_DTYPE)
        s[0] = x_p, 150., z_p, a_p, 1.45, 0.
        return lib.lmb_radial_intervals(
            _native.Grid(x0, 0., 0., nx, ny), nx * ny, s.ctypes.data, 1, k, 0.048,
            flags, aberration)
    assert intervals() > 0
    assert intervals(z_p=-200.) > 0
    assert intervals(z_p=0.75 / 0.048 + 2.1) > 0
    assert intervals(z_p=0.75 / 0.048 + 1.9) == 0   # too close
    assert intervals(z_p=5.) == 0                   # the plane cuts the sphere
    assert intervals(nx=3, ny=3) == 0               # too few pixels
    assert intervals(x0=-9000.) == 0                # too far
    assert intervals(flags=_native.LMB_BOHREN) == 0
    assert intervals(flags=cart | _native.LMB_FP64) > intervals()
    assert intervals(aberration=1e4) == 0
    assert intervals(aberration=20.) > 0
    assert intervals(z_p=np.nan) == 0 and intervals(x_p=np.inf) == 0
    assert intervals(k=50.) == 0
