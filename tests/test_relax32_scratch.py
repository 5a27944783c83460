"""The mixed form's relaxing reads the float-float splits of def and defp from
buffers that share an allocation with its own scratch.  What that allocation
holds besides depends on the schedule, the step does not: both schedules give
the same bits on every size, alone and after calls that leave other data there."""
import numpy as np
import pytest

from conftest import smooth_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 16, 32, 64])
def test_step_does_not_depend_on_the_schedule(mmh, fields, n):
    _, u = fields.initial_state(n, sigma=0.6, seed=90 + n)
    d, p = smooth_field(n, 0.2, 91 + n), smooth_field(n, 0.02, 92 + n)
    got = []
    for sched in (mmh.MMH_SCHED_TOL, mmh.MMH_SCHED_VCYCLE):
        with mmh.Context(n, precision=mmh.MMH_MIXED, schedule=sched) as ctx:
            for before in (None, "outputs", "smooth"):
                if before == "outputs":
                    ctx.defp2delta(d, np.zeros((n, n, n), order="F"), (n, n, n))
                elif before == "smooth":
                    ctx.nsmooth(p.copy(order="F"))
                v = u.copy(order="F")
                ctx.relaxing(v, d, p, 1.0, 1.0)
                got.append(v[0])
    assert np.isfinite(got[0]).all() and not np.array_equal(got[0], u[0])
    for g in got[1:]:
        assert np.array_equal(g, got[0])
