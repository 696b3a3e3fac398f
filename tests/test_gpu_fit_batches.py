'''GPU: a feature's fit from radial tables is the same to the bit alone, in
16 parts, and among others, in fewer: crops and pixel lists of more tiles
than the batches' parts.
'''
import numpy as np
import pytest

from pylorenzmie_b200 import _native

from tests.test_gpu_fit_radial import crops, fit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('side,listed,batches', [
    (201, False, (1, 2, 40, 64, 128, 256)), (151, True, (1, 3, 64, 128)),
    (301, False, (1, 20))])
def test_alone_and_among_others(side, listed, batches):
    items, starts = crops([(side, side)] * 4, seed=side)
    if listed:
        rng = np.random.default_rng(0)
        keep = np.sort(rng.choice(side * side, 9000, replace=False))
        items = [(d.ravel()[keep], None,
                  np.stack([keep % side, keep // side]).astype(float))
                 for d, _, _ in items]
    alone = [fit(items[i:i + 1], starts[i:i + 1], _native.LMB_FIT_RADIAL)
             for i in range(4)]
    for n in batches[1:]:
        pick = np.arange(n) % 4
        p, r = fit([items[i] for i in pick], starts[pick],
                   _native.LMB_FIT_RADIAL)
        for j, i in enumerate(pick):
            q, s = alone[i]
            assert np.array_equal(p[j], q[0]), (n, j)
            assert np.array_equal(r['dparams'][j], s['dparams'][0]), (n, j)
            assert r['nfev'][j] == s['nfev'][0]
