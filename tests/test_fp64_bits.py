"""The FP64 form's exact shortcuts (division by a shared reciprocal, scalings
and signs on the bits, integer minima) against the oracle bit for bit where
they leave the ordinary range: zero fields (zero numerators, zero speeds),
subnormal differences, values past the reciprocal's exponent range, spacings
that are no power of two, and limiter scales other than one."""
import numpy as np
import pytest

from conftest import smooth_field

pytestmark = pytest.mark.gpu
KINDS = ("smooth", "zero", "tiny", "subnormal", "rough", "huge")


def potential(n, kind, seed):
    if kind == "zero":
        return np.zeros((n, n, n), order="F")
    s = {"smooth": 0.3, "tiny": 1e-160, "subnormal": 3e-309, "rough": 2.0, "huge": 1e90}[kind]
    if kind == "rough":
        return np.asfortranarray(np.random.default_rng(seed).standard_normal((n, n, n)) * s)
    return smooth_field(n, s, seed)


def same(a, b):
    return np.array_equal(a, b, equal_nan=True) and np.array_equal(np.signbit(a)[~np.isnan(a)], np.signbit(b)[~np.isnan(b)])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,dx", [(8, 1.0), (16, 3.0), (16, 0.5)])
def test_metric(mmh, oracle, fields, n, dx, kind):
    _, u = fields.initial_state(n, sigma=0.8, seed=3)
    rho = np.asfortranarray(u[0])
    d = potential(n, kind, 4)
    with mmh.Context(n) as ctx:
        assert same(ctx.metric(d, rho, dx), oracle.metric(d, rho, dx))


@pytest.mark.parametrize("kd", KINDS)
@pytest.mark.parametrize("kp", ("smooth", "zero", "subnormal", "rough"))
def test_relaxing(mmh, oracle, fields, kd, kp):
    n = 16
    _, u = fields.initial_state(n, sigma=0.8, seed=5)
    d, p = potential(n, kd, 6), potential(n, kp, 7)
    ug = u.copy(order="F")
    uo = oracle.relaxing(u, d, p, 1.0)
    with mmh.Context(n) as ctx:
        ctx.relaxing(ug, d, p, 1.0, 1.0)
    uo = uo[0] if isinstance(uo, tuple) else uo
    assert same(ug[0], uo[0])


@pytest.mark.parametrize("kind", ("smooth", "zero", "rough"))
@pytest.mark.parametrize("dtold,dtaumesh", [(1.0, 1.0), (0.3, 7.0)])
def test_pass1(mmh, oracle, fields, kind, dtold, dtaumesh):
    n = 16
    _, u = fields.initial_state(n, sigma=0.8, seed=8)
    d = potential(n, kind, 9)
    t = np.asfortranarray(np.random.default_rng(1).standard_normal((n, n, n)) * 0.2)
    to, mxo, mco, do = oracle.limiter_pass1(t, d, u, dtold, dtaumesh)
    tg = t.copy(order="F")
    with mmh.Context(n) as ctx:
        mxg, mcg, dg = ctx.limiter_pass1(tg, d, np.asfortranarray(u[0]), dtold, dtaumesh)
    assert same(tg, to) and np.array_equal(mxo, mxg) and np.array_equal(mco, mcg)
    assert do["nexpand"] == dg["nexpand"] and do["detmin"] == dg["detmin"]


@pytest.mark.parametrize("kind", ("smooth", "zero", "tiny", "subnormal", "rough", "huge"))
@pytest.mark.parametrize("n", [8, 32])
def test_smooth(mmh, oracle, n, kind):
    a = potential(n, kind, 11)
    if kind == "huge":
        a = np.asfortranarray(a * 1e217)  # sums beyond the scaled form's range
    g = a.copy(order="F")
    with mmh.Context(n) as ctx:
        ctx.nsmooth(g)
        assert same(ctx.restrict(a), oracle.restrict(a))
    assert same(g, oracle.nsmooth(a))


@pytest.mark.parametrize("n", [4, 8, 16])
def test_zerosum_small(mmh, oracle, n):
    a = np.asfortranarray(np.random.default_rng(n).standard_normal((n, n, n)))
    g = a.copy(order="F")
    with mmh.Context(max(n, 8)) as ctx:
        ctx.zerosum(g)
    oracle.zerosum(a)
    assert same(g, a)


@pytest.mark.parametrize("n", [8, 16, 64, 128])
def test_smooth_passes(mmh, n):
    """The mixed form's three axis passes, in one launch up to 64^3, bit for
    bit: sums of two values and a fused multiply-add that only doubles."""
    a = np.random.default_rng(n).standard_normal((n, n, n))
    g = np.asfortranarray(a)
    with mmh.Context(n, precision=mmh.MMH_MIXED, schedule=mmh.MMH_SCHED_TOL) as ctx:
        ctx.nsmooth(g)
    for axis in range(3):
        a = 2.0 * a + (np.roll(a, 1, axis) + np.roll(a, -1, axis))
    assert same(g, a / 64)
