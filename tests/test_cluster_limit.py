"""Where no cluster of 16 CTAs fits, the small levels take smaller clusters or
their own launches, with the same bits: 16^3 FP64 sweeps by rows against the
oracle, and whole solves and iterations of every form against the same calls
with clusters of 16, on fresh contexts and after a change of the limit."""
import numpy as np
import pytest

from conftest import smooth_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sweeps,kind", [(1, "noise"), (2, "noise"), (9, "noise"), (3, "zero"), (2, "tiny")])
def test_rows_at_16(mmh, oracle, fields, sweeps, kind):
    n = 16
    _, u = fields.initial_state(n, sigma=0.8, seed=56)
    rho, defpot = np.asfortranarray(u[0]), smooth_field(n, 0.05, 57)
    s = {"noise": 1.0, "zero": 0.0, "tiny": 1e-290}[kind]
    rng = np.random.default_rng(sweeps)
    rhs, phi = (np.asfortranarray(rng.standard_normal((n, n, n)) * s) for _ in range(2))
    a, b = phi.copy(order="F"), phi.copy(order="F")
    oracle.relax(a, rhs, oracle.metric(defpot, rho, 4.0), 4.0, sweeps, 18, colour8=True)
    with mmh.Context(n) as ctx:
        ctx.max_cluster(8)
        ctx.relax(b, rhs, defpot, rho, 4.0, sweeps, 18)
    assert np.array_equal(a, b) and np.array_equal(np.signbit(a), np.signbit(b))


@pytest.mark.parametrize("form,n", [("mixed", 16), ("mixed", 32), ("mixed", 64), ("fp64", 16), ("fp64", 64),
                                    ("ref", 32), ("ref", 64)])
def test_same_bits(mmh, fields, form, n):
    rho = fields.lognormal_density(n, sigma=0.5, seed=70 + n).reshape((1, n, n, n), order="F")
    cfg = dict(precision=mmh.MMH_MIXED if form == "mixed" else mmh.MMH_FP64,
               schedule=mmh.MMH_SCHED_REF if form == "ref" else mmh.MMH_SCHED_TOL, tol=1e-9)

    def iterate(ctx):
        ctx.load(np.zeros((n, n, n), order="F"), rho)
        before = mmh.launch_count()
        d = ctx.iterate(2)
        launches = mmh.launch_count() - before
        got, u = np.zeros((n, n, n), order="F"), np.zeros((1, n, n, n), order="F")
        ctx.store(got, u)
        return got, u, d["vcycles"], launches

    with mmh.Context(n, **cfg) as ctx:
        iterate(ctx)  # the first sweeps on a size also time the tile shapes
        wide = iterate(ctx)
        ctx.max_cluster(8)
        narrow = [iterate(ctx)]
        ctx.max_cluster(16)
        back = iterate(ctx)
    with mmh.Context(n, **cfg) as ctx:
        ctx.max_cluster(8)
        narrow.append(iterate(ctx))
    for r in narrow + [back]:
        assert np.array_equal(r[0], wide[0]) and np.array_equal(r[1], wide[1]) and r[2] == wide[2]
    assert back[3] == wide[3]
    assert narrow[0][3] == narrow[1][3] and narrow[0][3] > wide[3]  # the other kernels ran


def test_limits_refused(mmh):
    with mmh.Context(8) as ctx:
        for ctas in (0, 4, 12, 32):
            with pytest.raises(mmh.MMHError):
                ctx.max_cluster(ctas)
