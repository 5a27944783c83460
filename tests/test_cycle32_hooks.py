"""The mixed form's levels of 32^3 and below while the timing hooks are armed:
they run launch by launch, so their launches are timed, and the solution, the
iteration counts and the residual have the bits of the one-launch cycle and
inner solve (the fields of a mesh already deformed, cycles of one to three
sweeps a side, the levels below a 64^3 grid and the solves on 32^3 and 16^3
themselves)."""
import numpy as np
import pytest

from conftest import smooth_field

pytestmark = pytest.mark.gpu


def problem(fields, n):
    _, u5 = fields.initial_state(n, sigma=0.6, seed=80 + n)
    rho = np.asfortranarray(u5[0])
    return smooth_field(n, 0.05, 81 + n), rho, np.asfortranarray(np.clip(1 - rho, -2, 2) / 30)


def solve(mmh, prob, n, kind=None, solves=1, **cfg):
    """Solutions and diagnostics of repeated solves on one context (the third
    replays the captured cycles), the hooks armed for `kind`, and their count."""
    defpot, rho, rhs0 = prob
    rho1 = np.asfortranarray(rho.reshape((1, n, n, n), order="F"))
    out, timed = [], None
    with mmh.Context(n, precision=mmh.MMH_MIXED, schedule=mmh.MMH_SCHED_TOL, **cfg) as ctx:
        if kind is not None:
            mmh.profile_start(kind)
        try:
            for _ in range(solves):
                u, rhs = np.zeros((n, n, n), order="F"), rhs0.copy(order="F")
                d = ctx.multigrid(u, rhs, defpot, rho1, 1.0, n, n, n, 1)
                out.append((u, d["vcycles"], d["resid_rel"]))
        finally:
            if kind is not None:
                timed = mmh.profile_stop()
    return out, timed


@pytest.mark.parametrize("n", [16, 32, 64])
@pytest.mark.parametrize("kind", ["K_GS", "K_RESIDUAL", "K_RESTRICT_RESID", "K_PROLONG"])
def test_small_levels_are_timed(mmh, fields, n, kind):
    prob = problem(fields, n)
    for level in (16, 32):
        if level > n:
            continue
        out, (launches, ms, cells) = solve(mmh, prob, n, getattr(mmh, kind) | mmh.K_F32 | mmh.K_AT(level), nu1=1,
                                           nu2=1, tol=1e-8)
        # at least one launch per cycle of each of these kinds
        assert launches >= out[0][1] > 0 and ms > 0 and cells > 0


@pytest.mark.parametrize("n,nu1,nu2,tol", [(16, 1, 1, 1e-8), (16, 2, 3, 1e-10), (16, 3, 1, 1e-12), (32, 1, 1, 1e-8),
                                           (32, 2, 2, 1e-10), (32, 1, 3, 1e-12), (32, 3, 2, 1e-9), (64, 1, 1, 1e-8),
                                           (64, 2, 2, 1e-10), (64, 3, 1, 1e-9)])
def test_same_bits(mmh, fields, n, nu1, nu2, tol):
    prob = problem(fields, n)
    cfg = dict(nu1=nu1, nu2=nu2, tol=tol)
    one, _ = solve(mmh, prob, n, solves=3, **cfg)
    per_level, _ = solve(mmh, prob, n, mmh.K_GS | mmh.K_F32, solves=1, **cfg)
    for u, its, rel in one:
        assert its == per_level[0][1] and rel == per_level[0][2]
        assert np.array_equal(u, per_level[0][0])
