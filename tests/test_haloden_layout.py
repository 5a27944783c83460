"""haloden on the two layouts of the positions, against the oracle bit for bit:
coordinates by rows (as they lie) and by particles; positions on and beyond the
box (the remainder's cases: below one period, one, two, more), wraps of the
search on the smallest and odd grids."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,ng,np_", [(4, 2, 1), (6, 3, 5), (14, 7, 40), (32, 16, 300), (93, 31, 900)])
def test_layouts(mmh, oracle, nf, ng, np_):
    rng = np.random.default_rng(ng)
    x = rng.uniform(0, nf * 0.999, (3, np_)).astype(np.float32)
    shift = rng.integers(-3, 4, (3, np_)) * np.float32(nf)
    x[:, ::2] += shift[:, ::2].astype(np.float32)
    x[0, 0] = np.float32(nf)  # one period exactly
    den, raw, wp = oracle.haloden(x, nf, ng)
    for xx in (x, np.asfortranarray(x)):
        d, r, w = mmh.haloden(xx, nf, ng)
        assert np.array_equal(r, raw) and np.array_equal(w, wp)
        assert np.allclose(d, den, rtol=2.0 ** -23, atol=0)
