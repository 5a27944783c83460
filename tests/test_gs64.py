"""The FP64 Gauss-Seidel kernels (box and row forms) against the oracle, bit
for bit: one sweep (prologue only), odd counts, counts past the point where a
4^3 grid stops changing, every size of the box form, the row form's row-block
sizes, and right-hand sides that take the plain division (zero, subnormal)."""
import numpy as np
import pytest

from conftest import smooth_field

pytestmark = pytest.mark.gpu


def problem(fields, n, seed):
    defpot, u = fields.initial_state(n, sigma=0.8, seed=seed)
    return smooth_field(n, 0.05, seed + 1), np.asfortranarray(u[0])


@pytest.mark.parametrize("n,sweeps,kind", [
    (4, 1, "noise"), (4, 7, "noise"), (4, 96, "smooth"), (4, 3, "zero"), (4, 3, "tiny"),
    (8, 1, "noise"), (8, 5, "noise"), (8, 3, "zero"), (16, 1, "noise"), (16, 9, "noise"), (16, 2, "tiny"),
    (32, 1, "noise"), (32, 3, "zero"), (64, 1, "noise"), (128, 2, "noise"), (256, 1, "noise")])
def test_sweeps_bitexact(mmh, oracle, fields, n, sweeps, kind):
    defpot, rho = problem(fields, n, 40 + n)
    rng = np.random.default_rng(n + sweeps)
    dx = 4.0 if n <= 16 else 1.0
    if kind == "smooth":  # a right-hand side without a mean: the sweeps settle
        rhs = smooth_field(n, 1.0, 9)
        rhs = np.asfortranarray(rhs - rhs.mean())
        phi = np.zeros((n, n, n), order="F")
    else:
        s = {"noise": 1.0, "zero": 0.0, "tiny": 1e-290}[kind]
        rhs = np.asfortranarray(rng.standard_normal((n, n, n)) * s)
        phi = np.asfortranarray(rng.standard_normal((n, n, n)) * s)
    a, b = phi.copy(order="F"), phi.copy(order="F")
    oracle.relax(a, rhs, oracle.metric(defpot, rho, dx), dx, sweeps, 18, colour8=True)
    with mmh.Context(max(n, 8)) as ctx:
        ctx.relax(b, rhs, defpot, rho, dx, sweeps, 18)
    assert np.array_equal(a, b)
    assert np.array_equal(np.signbit(a), np.signbit(b))
