"""The spectral outputs (transforms along single lines) against the packed
three-dimensional transform on noise, whose Nyquist planes are as large as any
other: every size has its own stages, and displacement and density also come
alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def packed_inverse(x):
    n = x.shape[0]
    m = n // 2
    rev = np.roll(x[::-1, ::-1], (1, 1), (0, 1))
    a, b = x[:, :, :m], np.conj(rev[:, :, ::-1][:, :, :m])
    z = np.fft.fftn(0.5 * (a + b) + 0.5j * np.exp(-2j * np.pi * np.arange(m) / n) * (a - b)) * (2.0 / n ** 3)
    return np.stack([z.real, z.imag], -1).reshape(n, n, n).transpose(2, 1, 0)


def outputs(d):
    n = d.shape[0]
    x = np.conj(np.fft.rfftn(d.transpose(2, 1, 0)))
    q = np.arange(n)
    q = np.where(q <= n // 2, q, q - n) * (2 * np.pi / n)
    k = [np.abs(q[: n // 2 + 1])[None, None, :], q[None, :, None], q[:, None, None]]
    return np.stack([packed_inverse(1j * w * x) for w in k], -1), packed_inverse(sum(w * w for w in k) * x)


@pytest.mark.parametrize("n", [8, 16, 32, 64, 128, 256, 512])
def test_outputs(mmh, n):
    rng = np.random.default_rng(n)
    d = np.asfortranarray(rng.standard_normal((n, n, n)))
    grad, delta = outputs(d)
    with mmh.Context(n) as ctx:
        g, e = np.zeros((n, n, n, 3), order="F"), np.zeros((n, n, n), order="F")
        ctx.scalar2gradient(d, g, (n, n, n))
        ctx.defp2delta(d, e, (n, n, n))
        # 2^-53 for each of the ~3 log2(n) roundings on the way to a value, and numpy's own
        tol = 6 * np.log2(n) * 2.0 ** -53
        assert np.linalg.norm(g - grad) <= tol * np.linalg.norm(grad)
        assert np.linalg.norm(e - delta) <= tol * np.linalg.norm(delta)
        ctx.load(d, np.asfortranarray(np.ones((1, n, n, n))))
        g2, e2 = np.zeros_like(g, order="F"), np.zeros_like(e, order="F")
        ctx.outputs(g2, e2)
    assert np.array_equal(g, g2) and np.array_equal(e, e2)
