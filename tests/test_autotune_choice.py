'''When the evaluation of a batch is timed, and what the timing decides: no
tuning is thrown away, and a stream is tuned on its first batch only.'''
import numpy as np
import pytest

from pylorenzmie_b200 import Instrument, _native, autotune
from pylorenzmie_b200.analysis import _fit

RADIAL = _native.LMB_FIT_RADIAL


@pytest.fixture
def tuned(monkeypatch):
    calls = []

    def tune(packed, starts, *args, reach=0, **kwargs):
        calls.append((len(starts), reach))
        return tune.answer
    tune.answer = 7
    monkeypatch.setattr(autotune, 'tune', tune)
    tune.calls = calls
    return tune


def evaluation(n, side, auto, z=200., aberration=0.):
    p = np.zeros((n, 6))
    p[:] = (side / 2., side / 2., z, 0.75, 1.45, 0.)
    packed = _fit.PackedFeatures(
        [(np.zeros((side, side), np.float32), (0., 0., side, side), None)] * n)
    cap = _fit.fit_capacity(p, 1.34, 0.447)
    return _fit.evaluation(packed, p, Instrument(), ('z_p',), cap, None, None,
                           auto, aberration)


@pytest.mark.parametrize('n,side', [(1, 201), (64, 51), (64, 201)])
def test_tables_are_not_tuned_unasked(tuned, n, side):
    for auto in (None, False):
        config, reach = evaluation(n, side, auto)
        assert config == RADIAL and reach > 0 and not tuned.calls


def test_asked_tuning_decides(tuned):
    assert evaluation(64, 201, True) == (7, 0)
    assert tuned.calls[0][1] > 0              # the tables are a candidate
    tuned.answer = RADIAL
    config, reach = evaluation(64, 201, True)
    assert config == RADIAL and reach == tuned.calls[1][1]


def test_without_tables(tuned):
    assert evaluation(64, 201, None, z=5.) == (7, 0)
    assert tuned.calls == [(64, 0)]
    assert evaluation(64, 201, False, z=5.) == (_fit.default_shape(64), 0)
    assert evaluation(1, 51, None) == (_fit.default_shape(1), 0)
    assert evaluation(64, 201, True, aberration=9.)[0] == RADIAL
    assert tuned.calls == [(64, 0)]


def test_keys_of_problem_classes():
    a = autotune.problem_key('B200', 30, 4000)
    assert autotune.problem_key('B200', 30, 4000, tables=True) != a


@pytest.mark.gpu
@pytest.mark.parametrize('auto', [None, True])
def test_stream_is_tuned_on_its_first_batch(tuned, auto):
    from pylorenzmie_b200 import Hologram, LorenzMie, Optimizer, workloads
    used = []
    run = _fit.fit_device

    def fit_device(*args, tile_config=0, **kwargs):
        used.append(tile_config)
        return run(*args, tile_config=tile_config, **kwargs)
    batches = []
    for n, z in ((64, 13.4), (64, 150.), (8, 150.), (64, 13.3)):
        p = np.zeros((n, 6))
        p[:] = (25., 25., z, 0.6, 1.45, 0.)
        m = LorenzMie(coordinates=LorenzMie.meshgrid((51, 51)),
                      particle=workloads.spheres(p[0])[0])
        h = m.hologram().reshape(51, 51)
        batches.append(([Hologram(h)] * n, p))
    opt = Optimizer(model=LorenzMie())
    opt.variables = ['x_p', 'y_p', 'z_p', 'a_p', 'n_p']
    _fit.fit_device = fit_device
    try:
        assert [len(d) for d in opt.optimize_stream(iter(batches),
                                                    autotune=auto)] == \
            [64, 64, 8, 64]
    finally:
        _fit.fit_device = run
    assert len(tuned.calls) == 1 and sorted(used) == sorted(
        [7, RADIAL, 7, 7] if auto is None else [7, 7, 7, 7])
