"""The rounding error of the spectral outputs, displacement and density, against
extended precision is no larger than that of three-dimensional transforms in
doubles: for a smooth potential, where the error of the high frequencies is
magnified most, and for noise."""
import numpy as np
import pytest
import scipy.fft

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(np.finfo(np.longdouble).eps > 2.0 ** -60, reason="long double is no wider than double")]


def outputs(d, real):
    """Displacement and density as the reference forms them (the packed inverse
    transform), in the precision `real`."""
    n = d.shape[0]
    m = n // 2
    two_pi = 8 * np.arctan(real(1))
    x = np.conj(scipy.fft.rfftn(np.ascontiguousarray(d.transpose(2, 1, 0)).astype(real)))
    q = np.arange(n)
    q = np.where(q <= m, q, q - n).astype(real) * (two_pi / n)
    k = [np.abs(q[: m + 1])[None, None, :], q[None, :, None], q[:, None, None]]
    angle = -two_pi * np.arange(m).astype(real) / n
    half = real(0.5)
    twiddle = half * 1j * (np.cos(angle) + 1j * np.sin(angle))

    def packed_inverse(y):
        rev = np.roll(y[::-1, ::-1], (1, 1), (0, 1))
        a, b = y[:, :, :m], np.conj(rev[:, :, ::-1][:, :, :m])
        z = scipy.fft.fftn(half * (a + b) + twiddle * (a - b)) * (real(2) / real(n) ** 3)
        return np.stack([z.real, z.imag], -1).reshape(n, n, n).transpose(2, 1, 0)

    return [packed_inverse(1j * w * x) for w in k] + [packed_inverse((k[0] ** 2 + k[1] ** 2 + k[2] ** 2) * x)]


def potential(n, kind):
    rng = np.random.default_rng(n)
    d = rng.standard_normal((n, n, n))
    if kind == "smooth":  # P(k) ~ k^-5.5, smoothed at 2 cells
        f = np.fft.fftfreq(n) * 2 * np.pi
        k2 = f[:, None, None] ** 2 + f[None, :, None] ** 2 + f[None, None, :] ** 2
        k2[0, 0, 0] = np.inf
        d = np.fft.ifftn(np.fft.fftn(d) * k2 ** -1.375 * np.exp(-2 * k2)).real
    return np.asfortranarray(d)


@pytest.mark.parametrize("kind", ["smooth", "noise"])
@pytest.mark.parametrize("n", [16, 32, 64])
def test_no_further_than_three_dimensional_transforms(mmh, n, kind):
    d = potential(n, kind)
    exact, plain = outputs(d, np.longdouble), outputs(d, np.float64)
    g, e = np.zeros((n, n, n, 3), order="F"), np.zeros((n, n, n), order="F")
    with mmh.Context(n) as ctx:
        ctx.scalar2gradient(d, g, (n, n, n))
        ctx.defp2delta(d, e, (n, n, n))
    mine = [g[..., 0], g[..., 1], g[..., 2], e]
    for field in (slice(0, 3), slice(3, 4)):
        error, other = (sum(float(((a - b) ** 2).sum()) for a, b in zip(x[field], exact[field])) for x in (mine, plain))
        assert error <= other
