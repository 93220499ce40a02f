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


def test_infinite_velocity_of_a_body_that_is_no_source_in_the_tree():
    # every other body's jerk stays finite in the tree's near field.  The tree is one leaf: an expansion would
    # hold this body's momentum, 0 times infinity.
    n = 3000
    x, y, z, vx, vy, vz, m = ics.plummer(n, 9)
    flags = np.full(n, 3, dtype=np.uint8)
    flags[7], vx[7] = 0, np.inf
    g = tcb.Gravity(p=4, ncrit=4096, variant=tcb.VARIANT_JERKS, direct_below=0)
    out = g.evaluate(x, y, z, m, vx, vy, vz, flags=flags)
    g.close()
    keep = flags == 3
    o = oracle.direct(x, y, z, np.where(keep, m, 0.0), np.where(keep, vx, 0.0), vy, vz,
                      targets=np.nonzero(keep)[0].astype(np.int32))
    for keys in (("ax", "ay", "az"), ("jx", "jy", "jz")):
        a, b = (np.stack(q) for q in zip(*[(out[k][keep], o[k]) for k in keys]))
        nb = np.linalg.norm(b, axis=0)
        assert (np.linalg.norm(a - b, axis=0) / np.maximum(nb, 1e-3 * np.sqrt(np.mean(nb ** 2)))).max() < 1e-11


def _root_errors(variant, r, softening=0.0):
    """|error| of the near field's 1 / sqrt(r^2 + eps^2) in units of the last place, and r^2 + eps^2: the
    potentials at distances r on the x axis of one body of mass 1 among massless ones, in a tree of one leaf."""
    x = np.concatenate([[0.0], r])
    n = len(x)
    zero = np.zeros(n)
    m = np.zeros(n)
    m[0] = 1.0
    g = tcb.Gravity(p=4, ncrit=n, variant=variant, direct_below=0, softening=softening)
    pot = g.evaluate(x, zero, zero, m, zero, zero, zero)["pot"][1:]
    g.close()
    q = r * r + softening * softening
    want = 1 / np.sqrt(q.astype(np.longdouble))
    return np.abs((pot - want) / np.spacing(want.astype(np.float64))).astype(np.float64), q


@pytest.mark.parametrize("variant", [tcb.VARIANT_TOP, tcb.VARIANT_JERKS])
@pytest.mark.parametrize("lo,hi", [(-20, 20), (-449, -440), (-460, -440), (-300, 100), (100, 200)])
def test_reciprocal_root_over_its_exponents(variant, lo, hi):
    # the library root's bound, 1 ulp.  The form used from 2^-900 to 2^900 stays inside it: half an ulp of its
    # last rounding, at most half of x y^2's, and 2^-8 ulp of the cut series; outside the library's is used.
    rng = np.random.default_rng(hi - lo)
    n = 4095
    r = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))
    r[:2] = np.ldexp(1.0, lo), np.nextafter(np.ldexp(1.0, hi), 0)
    err, _ = _root_errors(variant, r)
    assert err.max() <= 1.0 + 2.0 ** -8, err.max()


@pytest.mark.parametrize("variant", [tcb.VARIANT_TOP, tcb.VARIANT_JERKS])
@pytest.mark.parametrize("exponent", [-460, -451, -450, -449, 440, 449, 450, 451, 500])
def test_reciprocal_root_at_the_ends_of_its_range(variant, exponent):
    # a softening length puts r^2 + eps^2 on either side of the range's ends, whatever r is
    rng = np.random.default_rng(exponent + 1000)
    for f in (1.0, 1.1, 1.4142, 1.9):
        eps = float(np.ldexp(f, exponent))
        r = np.ldexp(rng.uniform(1.0, 2.0, 2047), rng.integers(*((-465, -440) if exponent < 0 else (100, 200)), 2047))
        err, q = _root_errors(variant, r, eps)
        assert err.max() <= 1.0 + 2.0 ** -8, (f, err.max())
