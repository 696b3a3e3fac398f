'''The recurrences of block_sphere_ab on the CPU, at the sizes where their
phases change and over drawn spheres: the waves inside, and the quotients
where these overflow, against extended precision.

Tolerance: 1e-11 of the largest coefficient and eps x, as the kernel's
(tests/test_gpu_mie_waves.py).
'''
import numpy as np
import pytest

from tests.cpu_harness.loader import Harness
from tests.test_gpu_mie_waves import LAMBDA, N_M, SPHERES, reference


@pytest.fixture(scope='module')
def h():
    return Harness()


def drawn():
    rng = np.random.default_rng(1)
    a = np.exp(rng.uniform(np.log(0.01), np.log(3.), 40))
    n = rng.uniform(0.5, 2.5, 40)
    k = np.where(rng.random(40) < 0.5, 0., rng.uniform(0., 0.1, 40))
    return list(zip(a, n, k))


@pytest.mark.parametrize('quotients', [False, True])
def test_against_extended_precision(h, quotients):
    for s in SPHERES + drawn():
        ab = h.sphere_ab(*s, N_M, LAMBDA, quotients=quotients)
        ref = reference(*s)
        assert ab.shape == ref.shape
        x = 2. * np.pi / LAMBDA * N_M * s[0]
        tol = 1e-11 * np.abs(ref).max() + 2.2e-16 * min(x, 1.)
        assert np.abs(ab - ref).max() <= tol, s


def test_tangents_of_both_ways(h):
    '''The waves' tangents are the quotients', to 1e-9 of the largest: n
    roundings of 1e-16 an order, times 1/|psi| up to 1e4.'''
    for s in SPHERES + drawn():
        d = [h.sphere_ab(*s, N_M, LAMBDA, deriv=True, quotients=q)[1]
             for q in (False, True)]
        scale = np.abs(d[1]).max()
        assert np.abs(d[0] - d[1]).max() <= 1e-9 * scale, s
