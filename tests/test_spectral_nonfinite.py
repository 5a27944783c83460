"""A cell of the potential that is not finite reaches every value of the
spectral outputs, as it does through a three-dimensional transform (every size
has its own stages; the first and last cell, one inside; both calls and each
output alone), and the next call on finite values is as on a fresh context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 16, 32, 64, 128, 256])
def test_nonfinite_cell_reaches_every_value(mmh, n):
    d = np.asfortranarray(np.random.default_rng(n).standard_normal((n, n, n)))
    with mmh.Context(n) as ctx:
        def outputs(a):
            g, e = np.zeros((n, n, n, 3), order="F"), np.zeros((n, n, n), order="F")
            ctx.scalar2gradient(a, g, (n, n, n))
            ctx.defp2delta(a, e, (n, n, n))
            return g, e

        g0, e0 = outputs(d)
        assert np.isfinite(g0).all() and np.isfinite(e0).all()
        cells = [((0, 0, 0), np.nan), ((n - 1,) * 3, np.inf), ((1, n // 2, 3), -np.inf)]
        for cell, bad in cells if n <= 64 else cells[2:]:
            b = d.copy(order="F")
            b[cell] = bad
            g, e = outputs(b)
            assert np.isnan(g).all() and np.isnan(e).all()
            ctx.load(b, np.asfortranarray(np.ones((1, n, n, n))))
            g, e = np.zeros_like(g0, order="F"), np.zeros_like(e0, order="F")
            ctx.outputs(g, e)
            assert np.isnan(g).all() and np.isnan(e).all()
            g, e = outputs(d)
            assert np.array_equal(g, g0) and np.array_equal(e, e0)
