'''Mie coefficients from the linear recurrences (lmb_mie.cuh) at the sizes
where their phases change: one to three orders, one short of, at and past a
warp's lanes and the block's threads, the largest capacity, and spheres whose
inside waves overflow FP64 and take the quotients' recurrence.'''
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_M, LAMBDA = 1.34, 0.447


def reference(a_p, n_p, k_p):
    '''a_n, b_n by the reference's recurrences (theory/Sphere.py:147-226) in
    extended precision.'''
    from oracle import mie as omie
    nmax = len(omie.mie_coefficients(a_p, n_p, k_p, N_M, LAMBDA)) - 1
    R, C = np.longdouble, np.clongdouble
    # the size parameter in FP64, as the kernel has it: what is compared is
    # the recurrences
    x = R(2. * np.pi / LAMBDA * N_M * a_p)
    m = C(complex(n_p / N_M, k_p / N_M))
    d, dm = np.zeros(nmax + 1, C), np.zeros(nmax + 1, R)
    for n in range(nmax, 0, -1):
        d[n - 1] = n / (m * x) - 1 / (d[n] + n / (m * x))
        dm[n - 1] = n / x - 1 / (dm[n] + n / x)
    i = C(1j)
    e = np.cos(x) + i * np.sin(x)
    psi, zeta, pz, d3 = np.sin(x), -i * e, (1 - e * e) / 2, i
    out = np.zeros((nmax + 1, 2), complex)
    for n in range(1, nmax + 1):
        t1, t3 = n / x - dm[n - 1], n / x - d3
        last = psi, zeta
        psi, zeta, pz = psi * t1, zeta * t3, pz * t1 * t3
        d3 = dm[n] + i / pz
        for j, f in enumerate((d[n] / m + n / x, d[n] * m + n / x)):
            out[n, j] = (f * psi - last[0]) / (f * zeta - last[1])
    return out


# a_p, n_p, k_p of 1, 2, 3, 7, 31, 32, 33, 62..65, 209 and 941 orders
SPHERES = [(0.0005, 1.5, 0.), (0.001, 1.5, 0.), (0.012, 1.5, 0.01), (0.1, 1.5, 0.),
           (1.0, 1.45, 0.), (1.05, 1.45, 0.), (1.09, 1.45, 0.), (2.45, 1.45, 0.),
           (2.5, 1.45, 0.02), (2.56, 1.45, 0.), (2.61, 1.45, 0.), (9.3, 1.6, 0.02),
           (47.78, 0.134, 0.), (47.78, 0.067, 0.)]


@pytest.mark.parametrize('spare', (0, 70))
def test_sphere_ab_edges(spare):
    '''Tolerance: n rounding errors of 1.1e-16 an order, times 1/|psi| where
    psi_n is close to a zero, 1e-4 at these sizes: 1e-11 for up to 1000
    orders.  Below one wave length psi_1's factor 1/x - D1_0 cancels to x, so
    that psi_1 is off by eps/x^2 of itself and a_1, b_1 of one order, which
    are differences of equal terms there, by eps x.  The tangents are the outputs' derivatives: central differences
    of step h = 1e-5 of the extended-precision reference, whose own error is
    the difference to those of step 2h, plus 1e-8.'''
    import torch
    from pylorenzmie_b200.theory import _kernels as K
    P = np.zeros((len(SPHERES), 6))
    P[:, 3:] = SPHERES
    refs = [reference(*s) for s in SPHERES]
    cap = max(len(r) for r in refs) - 1 + spare
    P = torch.as_tensor(P, device='cuda:0')
    ab, dab, nmax = K.sphere_ab(P, N_M, LAMBDA, cap, deriv=True)
    plain, none, _ = K.sphere_ab(P, N_M, LAMBDA, cap)
    assert none is None
    assert torch.equal(plain, ab)
    ab = ab.cpu().numpy().view(np.complex128)[..., 0]
    dab = dab.cpu().numpy().view(np.complex128)[..., 0]
    for i, ref in enumerate(refs):
        n = len(ref)
        assert int(nmax[i]) == n - 1
        x = 2. * np.pi / LAMBDA * N_M * SPHERES[i][0]
        tol = 1e-11 * np.abs(ref).max() + 2.2e-16 * min(x, 1.)
        assert np.abs(ab[i, :n] - ref).max() <= tol, SPHERES[i]
        assert not ab[i, n:].any() and not dab[i, n:].any()
        a_p, n_p, k_p = SPHERES[i]
        if a_p > 3.:
            continue    # n_max and sharp resonances move within the step
        h = 1e-5 * n_p
        diff = [(reference(a_p, n_p + s * h, k_p) - reference(a_p, n_p - s * h, k_p))
                / (2. * s * h) for s in (1, 2)]
        if any(len(d) != n for d in diff):
            continue
        tol = np.abs(diff[1] - diff[0]).max() + 1e-8 * np.abs(diff[0]).max()
        assert np.abs(dab[i, :n, 2:] - diff[0]).max() <= tol, SPHERES[i]
