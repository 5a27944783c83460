"""The one-launch cycle and inner solve of the mixed form on the levels of
32^3 and below: the solution meets its tolerance by the oracle's own residual,
equals the one of the per-level launches (which the guarded preconditioner
still takes) within the tolerance, and needs as many iterations."""
import numpy as np
import pytest

from conftest import smooth_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nu1,nu2,tol", [(16, 1, 1, 1e-8), (16, 2, 1, 1e-10), (32, 1, 1, 1e-8), (32, 1, 3, 1e-9),
                                           (32, 2, 2, 1e-12), (64, 1, 1, 1e-8), (128, 2, 2, 1e-10)])
def test_solve(mmh, oracle, fields, n, nu1, nu2, tol):
    _, u5 = fields.initial_state(n, sigma=0.6, seed=60 + n)
    rho = np.asfortranarray(u5[0])
    defpot = smooth_field(n, 0.05, 61 + n)
    rhs0 = np.asfortranarray(np.clip(1 - rho, -2, 2) / 30)
    sol, its = [], []
    for guards in (False, True):
        u, rhs = np.zeros((n, n, n), order="F"), rhs0.copy(order="F")
        with mmh.Context(n, precision=mmh.MMH_MIXED, schedule=mmh.MMH_SCHED_TOL, nu1=nu1, nu2=nu2, tol=tol,
                         precond_guards=guards) as ctx:
            before = mmh.launch_count()
            d = ctx.multigrid(u, rhs, defpot, np.asfortranarray(rho.reshape((1, n, n, n), order="F")), 1.0, n, n, n, 1)
            launches = mmh.launch_count() - before
        sol.append(u)
        its.append((d["vcycles"], launches))
        r = oracle.residual(u, rhs, oracle.metric(defpot, rho, 1.0), 1.0)
        # FP64 rounding of the oracle's residual: terms of n/(2 pi) |rhs|, 2^-52 each
        assert np.abs(r).max() <= (tol + 40 * n * 2.0 ** -52) * np.abs(rhs).max()
    assert its[0][0] <= its[1][0] + 2
    assert its[0][1] < its[1][1]
    # two solutions of relative residual tol differ by at most 2 tol |L^-1|: |L^-1| ~ n^2 / 40 / min(rho)
    assert np.abs(sol[0] - sol[1]).max() <= 2 * tol * n * n / 40 / rho.min() * np.abs(rhs).max()
