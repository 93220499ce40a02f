"""Values at the ends of the range in the near field and the time-step pass."""
import numpy as np
import pytest

import oracle
import taichi_collisional_b200 as tcb
from taichi_collisional_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [300, 2048])
@pytest.mark.parametrize("v", [np.inf, -np.inf, np.nan, 1e200])
def test_time_step_of_a_velocity_without_a_finite_square(n, v):
    # a pair whose relative speed is infinite has a step of zero, so both bodies' sums of 1 / tau^4 are
    # infinite; a NaN takes part in no comparison.  Finite sums: at most n FP64 terms of a few roundings each.
    x, y, z, vx, vy, vz, m = ics.plummer(n, 13)
    vx[5] = v
    g = tcb.Gravity(p=4, ncrit=16, theta=0.4, variant=tcb.VARIANT_TOP)
    out = g.evaluate_steps(x, y, z, m, vx, vy, vz, 0.025)
    g.close()
    o = oracle.evaluate_steps(x, y, z, m, vx, vy, vz, p=4, theta=0.4, ncrit=16, dt_param=0.025)
    a, b = out["timestep"], o["timestep"]
    assert np.array_equal(np.isinf(a), np.isinf(b)) and not np.isnan(a).any()
    assert np.isnan(v) or np.isinf(b).sum() > 1
    f = np.isfinite(b)
    np.testing.assert_allclose(a[f], b[f], rtol=1e-11)


def test_coincident_bodies_whose_velocities_differ_by_more_than_the_largest_double():
    # such a pair is left out like any other at r = 0.  All bodies lie in a plane and these velocities stand on
    # it, so every other pair's d . dv is 0 and its jerk m dv / r^3, at most some 1e299.
    n = 3000
    r = np.random.default_rng(17)
    x, y, z = np.zeros(n), r.uniform(-1, 1, n), r.uniform(-1, 1, n)
    v, m = np.zeros(n), np.full(n, 1e-20)
    y[1], z[1], v[0], v[1] = y[0], z[0], 1.2e308, -1.2e308
    g = tcb.Gravity(p=4, ncrit=4096, variant=tcb.VARIANT_JERKS, direct_below=0)
    out = g.evaluate(x, y, z, m, v, np.zeros(n), np.zeros(n))
    g.close()
    ry, rz = y[2:] - y[0], z[2:] - z[0]
    want = -1.2e308 * np.sum(1e-20 * (ry * ry + rz * rz) ** -1.5)
    assert abs(out["jx"][0] / want - 1) < 1e-11 and abs(out["jx"][1] / want + 1) < 1e-11
    assert all(np.isfinite(a).all() for a in out.values())
