'''GPU: the layout of the pixels belongs to the device copy of the
coordinates, whatever happens to the host array afterwards.'''
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('side', [64, 200])      # probed on the host, device
@pytest.mark.parametrize('first', ['jac', 'hologram'])
def test_host_array_changed_in_place(side, first):
    from pylorenzmie_b200 import LorenzMie, workloads
    p = np.zeros((8, 6))
    p[:, :2] = np.random.default_rng(0).uniform(0., side, (8, 2))
    p[:, 2:5] = 150., 0.75, 1.45
    spheres = workloads.spheres(p)
    c = np.vstack([LorenzMie.meshgrid((side, side)),
                   np.zeros((1, side * side))])
    want = LorenzMie(coordinates=c, particle=spheres).hologram()
    m = LorenzMie(coordinates=c, particle=spheres)
    if first == 'jac':
        m.particle = spheres[0]
        m.jac()                                  # makes the device copy
        m.particle = spheres
    else:
        m.hologram()
    m.coordinates[0] += 40.
    m.coordinates[2] += 20.
    assert np.array_equal(m.hologram(), want)
    m.coordinates = m.coordinates                # a new copy
    assert np.abs(m.hologram() - want).max() > 1e-3
