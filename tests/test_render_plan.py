'''The host side of lmb_render_plan and lmb_grid_probe_host (no GPU): errors,
the capacity of orders, the choice of tables, the workspace.'''
import numpy as np
import pytest

from pylorenzmie_b200 import LorenzMie, _native
from pylorenzmie_b200.theory import _kernels as K

K0 = 2. * np.pi / 0.447 * 1.34 * 0.048


def plan(rows, grid=(0., 0., 0., 300, 300), points=0, flags=3, npts=None,
         nitems=1):
    rec = np.array(rows, dtype=float).reshape(-1, 6).view(
        K.SPHERE_DTYPE).reshape(-1)
    g = None if grid is None else _native.Grid(*grid)
    p = _native.Render()
    npts = npts or (g.nx * g.ny if g else 90000)
    st = _native.load().lmb_render_plan(
        g, points, npts, rec.ctypes.data, len(rec), nitems, 1.34, 0.447, K0,
        0.048, flags, 0., p)
    return st, p


GOOD = [150., 150., 200., 0.75, 1.45, 0.]


def test_capacity_covers_the_largest_sphere():
    st, p = plan([GOOD, [0., 0., 300., 3., 1.6, 0.]])
    assert st == _native.LMB_OK
    want = K.wiscombe_yang([0.75, 3.], [1.45, 1.6], [0., 0.], 1.34, 0.447)
    assert p.nmax_cap == want.max() + 2


def test_invalid_spheres():
    for j in range(6):
        for v in (np.nan, np.inf):
            bad = list(GOOD)
            bad[j] = v
            assert plan([bad])[0] == _native.LMB_ERR_ARG
    for a, st in ((0., _native.LMB_ERR_ARG), (-1., _native.LMB_ERR_ARG),
                  (60., _native.LMB_ERR_NMAX), (1e300, _native.LMB_ERR_NMAX)):
        bad = list(GOOD)
        bad[3] = a
        assert plan([bad])[0] == st


@pytest.mark.parametrize('kwargs,tables', [
    ({}, True), ({'grid': None}, False), ({'flags': 7}, True),
    ({'flags': 7, 'points': 1}, False), ({'points': 1}, True),
    ({'flags': 2}, False), ({'grid': (0., 0., 0., 64, 64)}, False),
    ({'grid': (0., 0., 195., 300, 300)}, False)])
def test_choice_of_tables(kwargs, tables):
    st, p = plan([GOOD], **kwargs)
    assert st == _native.LMB_OK and (p.intervals > 0) == tables
    assert p.spheres == 0 and p.ab >= 48 + 8 and p.nmax > p.ab
    assert p.workspace_bytes >= p.tables >= p.nmax + 8
    assert (p.workspace_bytes > p.tables) == tables


def test_no_spheres():
    st, p = plan([], nitems=3)
    assert st == _native.LMB_OK and p.nmax_cap == 1 and p.intervals == 0


def test_probe_of_host_coordinates():
    c = np.vstack([LorenzMie.meshgrid((5, 7), corner=(1.5, 2.)),
                   np.zeros((1, 35))])
    g, full = K.make_grid(0., 35, K.probe_host(c))
    assert full and (g.x0, g.y0, g.nx, g.ny) == (1.5, 2., 7, 5)
    assert not K.make_grid(0., 34, K.probe_host(
        np.ascontiguousarray(c[:, :-1])))[1]
    c[2, 3] = 1.
    assert K.make_grid(0., 35, K.probe_host(c)) is None
