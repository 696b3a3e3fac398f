'''GPU: launches whose dynamic and static shared memory together pass the
48 KB that need no opt-in, while the dynamic part alone stays below.'''
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('cap', [61, 62, 63])
def test_layered_step_kernel_at_48_kb(cap):
    '''Three layers at 62 orders of capacity take 49 008 bytes of dynamic
    shared memory in the step kernel, which also declares static arrays.'''
    from pylorenzmie_b200 import Instrument, workloads
    from pylorenzmie_b200.analysis import _fit
    inst = Instrument()
    _, p, _, frac, idx = workloads.layered(1, seed=4)
    p[:, :4] = 50., 50., 200., 0.8
    particles = workloads.layered_spheres(p, frac, idx)
    data = workloads.render_particles(particles, [(101, 101)],
                                      instrument=inst)[0]
    packed = _fit.PackedFeatures([(data.ravel(), (0., 0., 101, 101), None)])
    start = p.copy()
    start[:, 2] += 2.
    params, res = _fit.fit_packed(
        packed, start, inst, ('x_p', 'y_p', 'z_p', 'a_p'), nmax_cap=cap,
        layers=_fit.layers_of(particles))
    assert res['status'][0] > 0
    assert abs(params[0, 2] - 200.) < 1.
