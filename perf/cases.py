'''The work that users of this package have it do, as timed cases.

Kinds of case (sizes from the package's own workloads and tests):

* ``hologram``  ``LorenzMie.hologram(device=True)``: one image of one or
  several spheres, from a small crop to a full camera frame; FP32 sums or
  ``double_precision``.
* ``field``     ``LorenzMie.field(device=True)``: the complex scattered
  field itself, for optical-force and propagation codes.
* ``batch``     ``LorenzMie.batch_hologram(device=True)``: many particle
  lists on one grid, as for training sets of neural networks.
* ``gradient``  ``theory.autograd.hologram`` forward and backward: the
  gradient of chi^2 with respect to sphere parameters in a torch program.
* ``fit``       ``Optimizer.optimize`` (one feature) and
  ``Optimizer.optimize_batch`` (many) on crops in host memory: equal or
  mixed sizes, homogeneous or three-layer spheres, ideal or aberrated optics.
* ``frame_fit`` ``Frame.optimize``: the features of one frame, each on its
  random tenth of the pixels.
* ``estimate``  ``Frame.estimate`` with the search on the device.

The fits' tables come back as 32-bit floats, as a program stores tracks:
the sums behind them are FP32 (the models' default).

The inputs are rendered by ``_Model`` below, plain torch in 64 bits, which
also gives the exact values.
'''
import math

import numpy as np
import torch

from pylorenzmie_b200 import Hologram, Instrument, LorenzMie, Optimizer, Sphere
from pylorenzmie_b200.analysis import Frame
from pylorenzmie_b200.theory import AberratedLorenzMie, LayeredSphere, autograd

WAVELENGTH, MAGNIFICATION, N_M, NOISE = 0.447, 0.048, 1.340, 0.003
KEYS = ('x_p', 'y_p', 'z_p', 'a_p', 'n_p', 'k_p')


def _fitted(case):
    '''The free parameters: of core-shell particles the material is known.'''
    return KEYS[:4] if case.get('layers', 1) > 1 else KEYS[:5]


def _table(case):
    return [k for v in _fitted(case) for k in (v, 'd' + v)] + [
        'success', 'npix', 'redchi']


def listed():
    return [
        # a small crop of one sphere: the call inside a user's own loop
        dict(name='hologram_64', kind='hologram', ny=64, nx=64, spheres=1,
             double=False),
        # a camera frame of 16 spheres
        dict(name='frame_16', kind='hologram', ny=1024, nx=1280, spheres=16,
             double=False),
        # the same call in 64 bits, on an odd frame of 5 spheres
        dict(name='frame_5_double', kind='hologram', ny=1023, nx=1279,
             spheres=5, double=True),
        # the complex field of a few spheres on a ragged grid
        dict(name='field_3', kind='field', ny=241, nx=319, spheres=3),
        # a training batch: 128 images of 4 spheres
        dict(name='batch_128x4', kind='batch', side=201, items=128, spheres=4),
        # gradients of large spheres, whose sums have the most orders
        dict(name='gradient_401', kind='gradient', side=401, items=12,
             a_lo=3., a_hi=6.),
        # one feature of default size, as in an interactive session
        dict(name='fit_1', kind='fit', features=1, lo=201, hi=201, layers=1,
             spherical=0.),
        # the features of several frames, equal crops
        dict(name='fit_256', kind='fit', features=256, lo=201, hi=201,
             layers=1, spherical=0.),
        # mixed crops, seen through an aberrated instrument
        dict(name='fit_48_mixed', kind='fit', features=48, lo=51, hi=301,
             layers=1, spherical=1.5),
        # core-shell particles followed from frame to frame
        dict(name='fit_24_layered', kind='fit', features=24, lo=151, hi=201,
             layers=3, spherical=0.),
        # one frame's features, each on a random tenth of its pixels
        dict(name='frame_fit_32', kind='frame_fit', features=32, side=121),
        # the global search of a frame's features
        dict(name='estimate_8', kind='estimate', features=8, side=121),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['hologram', 'hologram', 'field', 'batch', 'gradient',
                       'fit', 'fit', 'frame_fit', 'estimate'])
    if kind in ('hologram', 'field'):
        c = dict(kind=kind, ny=_log(rng, 48, 1024), nx=_log(rng, 48, 1280),
                 spheres=_log(rng, 1, 16))
        if kind == 'hologram':
            c['double'] = rng.random() < 0.3
        return c
    if kind == 'batch':
        return dict(kind=kind, side=_log(rng, 64, 201),
                    items=_log(rng, 4, 128), spheres=rng.randint(1, 4))
    if kind == 'gradient':
        a = rng.uniform(0.4, 4.)
        return dict(kind=kind, side=_log(rng, 51, 401),
                    items=_log(rng, 1, 12), a_lo=a, a_hi=1.5 * a)
    if kind == 'fit':
        layers = rng.choice([1, 1, 1, 3])
        lo = _log(rng, 51, 181) if layers == 1 else _log(rng, 131, 181)
        hi = min(int(lo * rng.uniform(1., 1.6)), 301 if layers == 1 else 201)
        n = _log(rng, 1, 128) if layers == 1 else _log(rng, 4, 24)
        s = rng.choice([0., 0., 1.5]) if layers == 1 else 0.
        return dict(kind=kind, features=n, lo=lo, hi=max(lo, hi),
                    layers=layers, spherical=s)
    if kind == 'frame_fit':
        return dict(kind=kind, features=_log(rng, 4, 32),
                    side=2 * rng.randint(40, 70) + 1)
    return dict(kind=kind, features=_log(rng, 2, 8),
                side=2 * rng.randint(40, 70) + 1)


# ---------------------------------------------------------------------------
# The inputs of a case, from its seed.

def _mid_order(a):
    '''Radii moved to the middle of the range that has their number of
    partial waves.  The count steps with the radius, chi^2 with it, and a
    minimum next to a step can lie on either side of it.'''
    k = 2. * np.pi / WAVELENGTH * N_M
    x = k * a
    for _ in range(20):
        c = x + 4.05 * np.cbrt(x)
        x -= (c - np.floor(c) - 0.5) * 0.9 / (1. + 1.35 * np.cbrt(x) ** -2)
    return x / k


def _scene(case, seed):
    '''Numbers of the case: sphere parameters and, for fits, starts.'''
    rng = np.random.default_rng([seed, 11])
    kind = case['kind']
    s = {}
    if kind in ('hologram', 'field'):
        n, ny, nx = case['spheres'], case['ny'], case['nx']
        p = np.zeros((n, 6))
        p[:, 0] = rng.uniform(0., nx, n)
        p[:, 1] = rng.uniform(0., ny, n)
        p[:, 3] = rng.uniform(0.4, 3.0, n)
        p[:, 4] = rng.uniform(1.38, 1.70, n)
        p[:, 5] = rng.uniform(0., 1e-3, n)
        p[:, 2] = np.maximum(rng.uniform(50., 600., n),
                             p[:, 3] / MAGNIFICATION + 10.)
        s['p'] = p
    elif kind == 'batch':
        n, side = case['items'] * case['spheres'], case['side']
        p = np.zeros((n, 6))
        p[:, :2] = rng.uniform(0., side, (n, 2))
        p[:, 2] = rng.uniform(100., 300., n)
        p[:, 3] = rng.uniform(0.4, 1.5, n)
        p[:, 4] = rng.uniform(1.38, 1.60, n)
        s['p'] = p
    elif kind == 'gradient':
        n, side = case['items'], case['side']
        p = np.zeros((n, 6))
        p[:, :2] = (side - 1) / 2. + rng.uniform(-2., 2., (n, 2))
        p[:, 3] = rng.uniform(case['a_lo'], case['a_hi'], n)
        p[:, 4] = rng.uniform(1.4, 1.8, n)
        p[:, 2] = np.maximum(rng.uniform(200., 600., n),
                             p[:, 3] / MAGNIFICATION + 40.)
        start = p.copy()
        start[:, :2] += rng.uniform(-0.3, 0.3, (n, 2))
        start[:, 2] += rng.uniform(-2., 2., n)
        start[:, 3] *= 1.01
        start[:, 4] += 0.003
        s['p'], s['start'] = p, start
    else:
        n = case['features']
        if kind == 'fit':
            sides = rng.integers(case['lo'], case['hi'] + 1, n)
        else:
            sides = np.full(n, case['side'])
        p = np.zeros((n, 6))
        c = (sides - 1) / 2.
        p[:, 0] = c + rng.uniform(-2., 2., n)
        p[:, 1] = c + rng.uniform(-2., 2., n)
        p[:, 2] = rng.uniform(150., 250., n)
        p[:, 3] = _mid_order(rng.uniform(0.6, 1.0, n))
        p[:, 4] = rng.uniform(1.40, 1.46, n)
        start = p.copy()
        start[:, 3] *= 1.03
        start[:, 4] += 0.01
        start[:, 2] += 5.
        if case.get('layers', 1) > 1:
            L = case['layers']
            p[:, 3] = start[:, 3] = _mid_order(rng.uniform(0.9, 1.5, n))
            p[:, 4] = rng.uniform(1.50, 1.60, n)
            inner = np.linspace(0.35, 0.6, L - 1)
            s['frac'] = inner + rng.uniform(-0.05, 0.05, (n, L - 1))
            s['core'] = rng.uniform(1.40, 1.45, (n, L - 1)).astype(complex)
            start[:, 3] *= 1.005
            start[:, 4] = p[:, 4]
            start[:, 2] = p[:, 2] + 1.
        s['p'], s['start'], s['sides'] = p, start, sides
    return s


def _grid(ny, nx, device):
    y, x = torch.meshgrid(torch.arange(ny, dtype=torch.float64, device=device),
                          torch.arange(nx, dtype=torch.float64, device=device),
                          indexing='ij')
    return x.reshape(-1), y.reshape(-1)


def _noise(shape, seed, device):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return NOISE * torch.randn(shape, generator=g, device=device,
                               dtype=torch.float64)


def _crops(case, s, seed, device):
    '''The fits' noisy crops: flat pixels with the feature they belong to.'''
    xs, ys, owner = [], [], []
    for i, side in enumerate(s['sides']):
        x, y = _grid(int(side), int(side), device)
        xs.append(x)
        ys.append(y)
        owner.append(torch.full((x.numel(),), i, device=device))
    x, y, owner = torch.cat(xs), torch.cat(ys), torch.cat(owner)
    m = _Model(x, y, owner, case.get('spherical', 0.), s.get('frac'),
               s.get('core'))
    clean = m.hologram(s['p'])
    return m, clean + _noise(clean.shape, seed, device)


def _frame(case, s, seed, device):
    '''One frame of well separated features on a grid of cells, each cell
    with its own feature's hologram, and the features' boxes.'''
    n, side = case['features'], case['side']
    cols, rows, pitch = min(n, 8), -(-n // min(n, 8)), side + 30
    corner = np.stack([15 + pitch * (np.arange(n) % cols),
                       15 + pitch * (np.arange(n) // cols)], axis=1)
    p, start = s['p'].copy(), s['start'].copy()
    x, y = _grid(pitch, pitch, device)
    data = torch.ones((rows, cols, pitch, pitch), dtype=torch.float64,
                      device=device)
    for i in range(n):
        data[i // cols, i % cols] = _Model(x - 15., y - 15.).hologram(
            p[i][None]).reshape(pitch, pitch)
    data = data.transpose(1, 2).reshape(rows * pitch, cols * pitch)
    data = data + _noise(data.shape, seed, device)
    start[:, :2] += corner
    boxes = [((int(cx), int(cy)), side, side) for cx, cy in corner]
    return start, data.cpu().numpy(), boxes


def _sphere(row):
    s = Sphere(a_p=row[3], n_p=row[4], k_p=row[5])
    s.r_p = row[:3]
    return s


def _instrument():
    return Instrument(wavelength=WAVELENGTH, magnification=MAGNIFICATION,
                      n_m=N_M, noise=NOISE)


def prepare(case, seed):
    dev = torch.device('cuda')
    s = _scene(case, seed)
    kind = case['kind']
    state = {'case': case, 'scene': s}
    if kind in ('hologram', 'field', 'batch'):
        shape = ((case['side'],) * 2 if kind == 'batch' else
                 (case['ny'], case['nx']))
        model = LorenzMie(coordinates=LorenzMie.meshgrid(shape),
                          instrument=_instrument(),
                          double_precision=case.get('double', False))
        spheres = [_sphere(row) for row in s['p']]
        if kind == 'batch':
            k = case['spheres']
            state['lists'] = [spheres[i:i + k]
                              for i in range(0, len(spheres), k)]
        else:
            model.particle = spheres if len(spheres) > 1 else spheres[0]
        state['model'] = model
    elif kind == 'gradient':
        x, y = _grid(case['side'], case['side'], dev)
        state['coords'] = torch.stack([x, y])
        data = torch.stack([_Model(x, y).hologram(row[None])
                            for row in s['p']])
        state['data'] = (data + _noise(data.shape, seed, dev)).float()
        state['params'] = torch.tensor(s['start'], dtype=torch.float32,
                                       device=dev, requires_grad=True)
        state['instrument'] = _instrument()
    elif kind == 'fit':
        _, data = _crops(case, s, seed, dev)
        data = data.cpu().numpy()
        state['holograms'], at = [], 0
        for side in s['sides']:
            n = int(side) ** 2
            state['holograms'].append(Hologram(
                data[at:at + n].reshape(side, side).copy()))
            at += n
        if case['spherical']:
            model = AberratedLorenzMie(instrument=_instrument(),
                                       spherical=case['spherical'])
        else:
            model = LorenzMie(instrument=_instrument())
        opt = Optimizer(model=model)
        opt.variables = list(_fitted(case))
        state['optimizer'] = opt
    else:
        start, data, boxes = _frame(case, s, seed, dev)
        frame = Frame(instrument=_instrument())
        frame.data = data
        frame.bboxes = boxes
        for i, f in enumerate(frame.features):
            f.estimator.seed = 1000 + i
            f.estimator.device_search = True
        state['frame'], state['start'] = frame, start
        state['seed'] = seed
    return state


def _columns(table, names):
    out = {}
    for name in names:
        v = np.asarray(table[name])
        out[name] = v.astype(np.float32) if v.dtype.kind == 'f' else v
    return out


def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'hologram':
        return state['model'].hologram(device=True)
    if kind == 'field':
        return state['model'].field(device=True)
    if kind == 'batch':
        return state['model'].batch_hologram(state['lists'], device=True)
    if kind == 'gradient':
        params = state['params']
        h = autograd.hologram(params, state['coords'], state['instrument'])
        chi2 = ((h - state['data']) * (1. / NOISE)).square().sum()
        grad, = torch.autograd.grad(chi2, params)
        return {'hologram': h.detach(), 'grad': grad}
    if kind == 'fit':
        opt, s = state['optimizer'], state['scene']
        if case['features'] == 1 and case['layers'] == 1:
            opt.model.particle = _sphere(s['start'][0])
            result = opt.optimize(state['holograms'][0])
            return {k: (np.float32(result[k]) if isinstance(
                result[k], float) else int(result[k])) for k in _table(case)}
        if case['layers'] > 1:
            particles = []
            for row, f, c in zip(s['start'], s['frac'], s['core']):
                p = LayeredSphere(a_p=row[3], n_p=row[4], k_p=row[5],
                                  fractions=tuple(f), core_indices=tuple(c))
                p.r_p = row[:3]
                particles.append(p)
            table = opt.optimize_batch(state['holograms'], particles)
        else:
            table = opt.optimize_batch(state['holograms'], starts=s['start'])
        return _columns(table, _table(case))
    frame = state['frame']
    np.random.seed(state['seed'] % (1 << 31))   # the random pixel subsets
    if kind == 'frame_fit':
        for f, row in zip(frame.features, state['start']):
            f.particle.r_p = row[:3]
            f.particle.a_p, f.particle.n_p = row[3], row[4]
        return _columns(frame.optimize(), _table(case))
    frame.estimate()
    return np.array([[f.particle.z_p, f.particle.a_p, f.particle.n_p]
                     for f in frame.features])


def work(case):
    '''Bytes: inputs and outputs once.  Operations: 70 per pixel and
    particle (phase, projection, superposition), 200 with the derivatives,
    and for a fit three evaluations, fewer than any fit here needs.'''
    kind = case['kind']
    if kind in ('hologram', 'field', 'batch'):
        npts = case['side'] ** 2 if kind == 'batch' else case['ny'] * case['nx']
        items = case.get('items', 1)
        out = 24 if kind == 'field' else 8 if case.get('double') else 4
        return {'bytes': npts * (16 + items * out),
                'flops': 70 * npts * items * case['spheres']}
    if kind == 'gradient':
        n = case['side'] ** 2 * case['items']
        return {'bytes': 16 * case['side'] ** 2 + 12 * n, 'flops': 270 * n}
    if kind == 'fit':
        n = case['features'] * (case['lo'] ** 2 + case['hi'] ** 2) // 2
        return {'bytes': 8 * n, 'flops': 3 * 200 * n}
    n = case['features'] * case['side'] ** 2
    if kind == 'frame_fit':
        return {'bytes': 8 * n, 'flops': 3 * 200 * n // 10}
    # 30 candidates of each feature, 20 generations, a fiftieth of the pixels
    return {'bytes': 8 * n, 'flops': 70 * 600 * n // 50}


# ---------------------------------------------------------------------------
# The exact values: numpy for the coefficients, torch for the pixels, all in
# 64 bits.

def _orders(x, m):
    '''Partial waves of layered spheres, x and m (n, L).'''
    xl = x[:, -1]
    ns = np.where(xl <= 8., np.floor(xl + 4. * np.cbrt(xl) + 1.),
                  np.floor(xl + 4.05 * np.cbrt(xl) + 2.))
    return np.maximum(ns, np.maximum(
        np.abs(x * m).max(axis=1),
        np.abs(np.roll(x, -1, axis=1) * m).max(axis=1))).astype(int)


def _d1(z, nmax, start):
    '''Logarithmic derivatives (top + 1, n), zero from order start on.'''
    top = int(start.max())
    d = np.zeros((top + 2, z.size), complex)
    for n in range(top, 0, -1):
        d[n - 1] = np.where(n > start, 0., n / z - 1. / (d[n] + n / z))
    return d


def _upward(z, d1, top):
    '''psi, zeta and D3 (top + 1, n).'''
    psi, zeta, d3 = (np.zeros((top + 1, z.size), complex) for _ in range(3))
    psi[0], zeta[0], d3[0] = np.sin(z), -1j * np.exp(1j * z), 1j
    pz = 0.5 * (1. - np.exp(2j * z))
    for n in range(1, top + 1):
        t1, t3 = n / z - d1[n - 1], n / z - d3[n - 1]
        psi[n], zeta[n] = psi[n - 1] * t1, zeta[n - 1] * t3
        pz = pz * t1 * t3
        d3[n] = d1[n] + 1j / pz
    return psi, zeta, d3


def _coefficients(radii, indices):
    '''a_n, b_n (n, top + 1, 2) and the orders of spheres given by radii
    (n, L) and complex indices (n, L), core first.'''
    with np.errstate(all='ignore'):
        k = 2. * np.pi / WAVELENGTH * N_M
        x, m = k * radii, indices / N_M
        L = x.shape[1]
        nmax = _orders(x, m)
        top = int(nmax.max())
        start = nmax + (1 if L > 1 else 0)
        ha = _d1(x[:, 0] * m[:, 0], nmax, start)[:top + 1]
        hb = ha
        for i in range(1, L):
            z1, z2 = x[:, i] * m[:, i], x[:, i - 1] * m[:, i]
            da, db = _d1(z1, nmax, start), _d1(z2, nmax, start)
            ea, eb = _upward(z1, da, top)[2], _upward(z2, db, top)[2]
            q = (np.exp(-2j * z2) - 1.) / (np.exp(-2j * z1) - 1.)
            na, nb = np.zeros_like(ha), np.zeros_like(ha)
            for n in range(1, top + 1):
                q = q * (x[:, i - 1] / x[:, i]) ** 2 * \
                    (z1 * da[n] + n) * (n - z1 * ea[n - 1]) / \
                    ((z2 * db[n] + n) * (n - z2 * eb[n - 1]))
                for old, new, u, v in ((ha, na, m[:, i], m[:, i - 1]),
                                       (hb, nb, m[:, i - 1], m[:, i])):
                    g1, g2 = u * old[n] - v * db[n], u * old[n] - v * eb[n]
                    new[n] = (g2 * da[n] - q * g1 * ea[n]) / (g2 - q * g1)
            ha, hb = na, nb
        xl, ml = x[:, -1], m[:, -1]
        z = xl.astype(complex)
        psi, zeta, _ = _upward(z, _d1(z, nmax, nmax), top)
        ab = np.zeros((top + 1, x.shape[0], 2), complex)
        for n in range(1, top + 1):
            for j, f in ((0, ha[n] / ml + n / xl), (1, hb[n] * ml + n / xl)):
                ab[n, :, j] = (f * psi[n] - psi[n - 1]) / \
                    (f * zeta[n] - zeta[n - 1])
        ab[np.arange(top + 1)[:, None] > nmax[None]] = 0.
    return ab, nmax


def _intensity(e):
    return ((e[0] + 1.).abs().square() + e[1].abs().square() +
            e[2].abs().square())


class _Model:
    '''Fields and holograms of one sphere per owner, at flat pixels of the
    plane z = 0 (owner: the row of the parameters each pixel belongs to).'''

    def __init__(self, x, y, owner=None, spherical=0., frac=None, core=None):
        self.x, self.y, self.owner = x, y, owner
        self.spherical, self.frac, self.core = spherical, frac, core

    def field(self, p):
        dev = self.x.device
        radii, index = p[:, 3:4], p[:, 4:5] + 1j * p[:, 5:6]
        if self.frac is not None:
            radii = np.concatenate([self.frac * radii, radii], axis=1)
            index = np.concatenate([self.core, index], axis=1)
        ab, _ = _coefficients(radii, index)
        ab = torch.from_numpy(ab).to(dev)
        pt = torch.from_numpy(np.ascontiguousarray(p)).to(dev)
        own = self.owner

        def spread(v):
            return v[0] if own is None else v[own]
        k = 2. * np.pi / WAVELENGTH * N_M * MAGNIFICATION
        kx = k * (self.x - spread(pt[:, 0]))
        ky = k * (self.y - spread(pt[:, 1]))
        zp = spread(pt[:, 2])
        kz = (k * zp).expand_as(kx)
        krho = torch.hypot(kx, ky)
        kr = torch.hypot(krho, kz)
        one = krho == 0.
        safe = torch.where(one, 1., krho)
        cp, sp = torch.where(one, 1., kx / safe), ky / safe
        ct, st = kz / kr, krho / kr
        # e^{i (kr - kz)}: the sums below leave out e^{i kr}
        phase = torch.polar(torch.ones_like(kr), krho * krho / (kr + kz))
        h2 = torch.ones_like(kr).to(torch.complex128)
        h1 = -1j * h2
        pi1, pi = torch.zeros_like(kr), torch.ones_like(kr)
        s0, s1, s2 = (torch.zeros_like(h2) for _ in range(3))
        fac = 1. + 0j
        for n in range(1, ab.shape[0]):
            sw = pi * ct
            tw = sw - pi1
            tau = pi1 - n * tw
            h = (2. * n - 1.) / kr * h1 - h2
            d = n / kr * h - h1
            fac *= 1j
            en = fac * (2. * n + 1.) / (n * n + n)
            a = 1j * en * spread(ab[n, :, 0])
            b = en * spread(ab[n, :, 1])
            s0 += (n * n + n) * a * (pi * h)
            ad, bh = a * d, b * h
            s1 += tau * ad - pi * bh
            s2 += pi * ad - tau * bh
            pi1, pi = pi, sw + (1. + 1. / n) * tw
            h2, h1 = h1, h
        e0, e1, e2 = (cp * st / (kr * kr)) * s0, (cp / kr) * s1, (sp / kr) * s2
        if self.spherical:
            rsq = krho * krho / (k * k)
            q = rsq / (rsq + zp * zp)
            phi = 4. * N_M ** 3 / k * self.spherical * q * q
            phase = phase * torch.polar(torch.ones_like(phi), phi)
        return torch.stack([
            phase * (st * cp * e0 + ct * cp * e1 - sp * e2),
            phase * (st * sp * e0 + ct * sp * e1 + cp * e2),
            phase * (ct * e0 - st * e1)])

    def hologram(self, p):
        return _intensity(self.field(p))

    def slopes(self, p, columns):
        '''Central differences of the hologram, (len(columns), npix).'''
        out = []
        for j in columns:
            step = 1e-4 if j < 3 else 1e-8
            hi, lo = p.copy(), p.copy()
            hi[:, j] += step
            lo[:, j] -= step
            out.append((self.hologram(hi) - self.hologram(lo)) / (2. * step))
        return torch.stack(out)


def _exact_fit(m, data, start, fitted):
    '''The least-squares minimum from ``start`` and its statistics.'''
    p = start.copy()
    n, nv = p.shape[0], len(fitted)
    own = m.owner
    npix = torch.bincount(own, minlength=n).double()

    def sums(v):
        return torch.zeros(n, dtype=torch.float64, device=v.device
                           ).index_add_(0, own, v)
    for step in range(8):
        r = (m.hologram(p) - data) / NOISE
        J = m.slopes(p, range(nv)) / NOISE
        A = torch.stack([torch.stack([sums(J[i] * J[j]) for j in range(nv)],
                                     -1) for i in range(nv)], -2)
        if step == 7:
            break
        g = torch.stack([sums(J[i] * r) for i in range(nv)], -1)
        p[:, :nv] -= torch.linalg.solve(A, g).cpu().numpy()
    redchi = sums(r * r) / (npix - nv)
    err = (redchi[:, None] * torch.linalg.inv(A).diagonal(
        dim1=-2, dim2=-1)).sqrt()
    out = {}
    for j, v in enumerate(fitted):
        out[v], out['d' + v] = p[:, j].copy(), err[:, j].cpu().numpy()
    out['success'] = out['npix'] = None
    out['redchi'] = redchi.cpu().numpy()
    return out


def exact(case, seed):
    dev = torch.device('cuda')
    s = _scene(case, seed)
    kind = case['kind']
    if kind in ('hologram', 'field'):
        m = _Model(*_grid(case['ny'], case['nx'], dev))
        e = 0.
        for row in s['p']:
            e = e + m.field(row[None])
        return e if kind == 'field' else _intensity(e)
    if kind == 'batch':
        m = _Model(*_grid(case['side'], case['side'], dev))
        k = case['spheres']
        out = []
        for i in range(case['items']):
            e = 0.
            for row in s['p'][i * k:(i + 1) * k]:
                e = e + m.field(row[None])
            out.append(_intensity(e))
        return torch.stack(out)
    if kind == 'gradient':
        state = prepare(case, seed)
        start = state['params'].detach().double().cpu().numpy()
        m = _Model(*_grid(case['side'], case['side'], dev))
        h = torch.stack([m.hologram(row[None]) for row in start])
        r = 2. * (h - state['data'].double()) / NOISE ** 2
        grad = torch.stack([(m.slopes(row[None], range(6)) * ri).sum(-1)
                            for row, ri in zip(start, r)])
        return {'hologram': h, 'grad': grad}
    if kind == 'fit' and case['features'] * case['hi'] ** 2 <= 3_000_000:
        m, data = _crops(case, s, seed, dev)
        out = _exact_fit(m, data, s['start'], _fitted(case))
        if case['features'] == 1 and case['layers'] == 1:
            out = {k: None if v is None else float(v[0])
                   for k, v in out.items()}
        return out
    return None
