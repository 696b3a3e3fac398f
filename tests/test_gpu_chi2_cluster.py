'''The population chi^2 where an item's blocks of 128 pixels fit one cluster of
eight and add their sums themselves, and one past it: against the FP64 oracle,
and bit-identical between the two where a larger crop shares the launch.'''
import numpy as np
import pytest

from oracle import field as ofield

pytestmark = pytest.mark.gpu

KEYS = ('x_p', 'y_p', 'z_p', 'a_p', 'n_p', 'k_p')


@pytest.mark.parametrize('npix', (1, 127, 128, 129, 300, 1023, 1024, 1025, 1300))
def test_chi2_blocks(npix):
    '''Tolerance: a hologram off by e moves chi^2 by 2 e / noise sum |r|; e is
    2e-5 in FP32 and 1e-12 in FP64.'''
    import torch
    from pylorenzmie_b200.theory import _kernels as K
    rng = np.random.default_rng(npix)
    coords = ofield.meshgrid((41, 53))
    coords = coords[:, np.sort(rng.permutation(coords.shape[1])[:npix])]
    inst = ofield.DEFAULT_INSTRUMENT
    S = 5
    P = np.tile([20.2, 25.9, 140., 0.8, 1.45, 0.], (S, 1))
    P[:, 2] = rng.uniform(100., 300., S)
    P[:, 3] = rng.uniform(0.3, 2.0, S)
    data = 1. + rng.normal(0., 0.2, npix)
    if npix > 200:
        data[130] = np.nan        # skipped, as numpy.nansum does
    r = np.array([(ofield.hologram(coords, [dict(zip(KEYS, p))], inst) - data) / 0.05
                  for p in P])
    ref, size = np.nansum(r * r, axis=1), np.nansum(np.abs(r), axis=1)
    dev = torch.device('cuda')
    c3 = torch.from_numpy(np.vstack([coords, np.zeros(npix)])).to(dev)
    d = torch.from_numpy(data).to(dev)
    rec = np.zeros(S, dtype=K.SPHERE_DTYPE)
    for j, key in enumerate(KEYS):
        rec[key] = P[:, j]
    sp = K.spheres_tensor(rec, dev)
    cap = K.nmax_cap_for(P[:, 3], P[:, 4], P[:, 5], 1.34, 0.447)
    ab, _, nmax = K.sphere_ab(sp, 1.34, 0.447, cap)
    item_start = torch.arange(S + 1, dtype=torch.int32, device=dev)
    k = ofield.wavenumber(1.34, 0.447, 0.048)
    for fp64 in (True, False):
        got, bad = K.chi2(c3, d, 0.05, sp, item_start, ab, nmax, cap, k,
                          fp64=fp64, nonfinite=True)
        assert not bad.any()
        off = np.abs(got.cpu().numpy() - ref)
        assert np.all(off <= 2. * (1e-12 if fp64 else 2e-5) / 0.05 * size), off
        # the same crop beside one of 2000 pixels, which takes the other way
        pad = torch.zeros((3, 2000), dtype=torch.float64, device=dev)
        start = torch.tensor([0, npix, npix + 2000], dtype=torch.int64, device=dev)
        crop = torch.zeros(S, dtype=torch.int32, device=dev)
        both = K.chi2_crops(torch.cat([c3, pad], 1), torch.cat([d, pad[0]]), 0.05,
                            start, crop, 2000, sp, item_start, ab, nmax, cap, k,
                            fp64=fp64)[0]
        assert torch.equal(both, got)
