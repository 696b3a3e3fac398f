'''Sizes that do not fit one another are refused before anything is launched
(no GPU): the grid's pixels and npts, the plan's counts and the call's.'''
import ctypes

import numpy as np
import pytest

from pylorenzmie_b200 import _native

K0 = 2. * np.pi / 0.447 * 1.34 * 0.048
GRID = _native.Grid(0., 0., 0., 300, 300)
HERE = ctypes.create_string_buffer(64)      # a pointer that is never read
AT = ctypes.addressof(HERE)


def spheres(n):
    rec = np.zeros(n, dtype=_native.SPHERE_DTYPE)
    rec[:] = (150., 150., 200., 0.75, 1.45, 0.)
    return rec


def plan(npts=90000, n=2, nitems=1):
    rec, p = spheres(n), _native.Render()
    st = _native.load().lmb_render_plan(
        GRID, 0, npts, rec.ctypes.data, n, nitems, 1.34, 0.447, K0, 0.048, 3,
        0., p)
    return st, p


def run(p, npts=90000, n=2, start=(0, 2)):
    rec, s = spheres(n), np.array(start, dtype=np.int32)
    return _native.load().lmb_render_run(
        p, GRID, 0, AT, npts, rec.ctypes.data, n, s.ctypes.data, len(s) - 1,
        1.34, 0.447, K0, 3, 0., 0, AT, AT, p.workspace_bytes, None)


@pytest.mark.parametrize('npts', [1, 89999, 90001, 89700])
def test_grid_and_npts(npts):
    lib = _native.load()
    assert plan(npts=npts)[0] == _native.LMB_ERR_ARG
    nbytes = lib.lmb_radial_workspace_bytes(1, 400, 3)
    for fn in (lib.lmb_hologram_grid, lib.lmb_field_grid):
        assert fn(GRID, None, npts, AT, AT, 1, 1, 400, AT, AT, 30, K0, 3, 0.,
                  AT, AT, nbytes, None) == _native.LMB_ERR_ARG


@pytest.mark.parametrize('kwargs', [
    {'n': 3, 'start': (0, 3)}, {'n': 1, 'start': (0, 1)},
    {'start': (0, 1, 2)}, {'npts': 90300}, {'npts': 45000},
    {'start': (0, 3)}, {'start': (-1, 2)}])
def test_a_call_other_than_the_plan(kwargs):
    st, p = plan()
    assert st == _native.LMB_OK
    assert run(p, **kwargs) == _native.LMB_ERR_ARG


def test_offsets_that_descend():
    st, p = plan(nitems=2)
    assert st == _native.LMB_OK
    assert run(p, start=(0, 2, 1)) == _native.LMB_ERR_ARG
