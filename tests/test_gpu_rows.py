"""Near-field work items, the time-step pass and the direct sums at the edges of their kernels.

Tolerance: every value is a sum of at most n = 5,000 FP64 terms in another order than the oracle's;
the terms carry a few roundings each, so a relative difference of (n + 10) 2^-53 of the sum of the
terms' magnitudes, 5.6e-13, bounds it.  The field of a centrally concentrated cluster is about that
sum over ten, and bodies whose field cancels are measured against 1e-3 of the rms: 1e-11."""
import numpy as np
import pytest

import oracle
import taichi_collisional_b200 as tcb
from taichi_collisional_b200 import ics

pytestmark = pytest.mark.gpu
ACC, JERK = ("ax", "ay", "az"), ("jx", "jy", "jz")


def _close(out, ref, keys, sel=slice(None)):
    a = np.stack([out[k][sel] for k in keys])
    b = np.stack([ref[k][sel] for k in keys])
    nb = np.linalg.norm(b, axis=0)
    err = np.linalg.norm(a - b, axis=0) / np.maximum(nb, 1e-3 * np.sqrt(np.mean(nb ** 2)))
    assert err.max() < 1e-11, (keys, err.max())


def _cluster(n, seed):
    """A Plummer sphere with three far bodies, whose leaves have nearly every body as a source."""
    b = [np.array(a) for a in ics.plummer(n, seed)]
    for k in range(3):
        b[k][k] += 40.0 + 7 * k
    return b


@pytest.mark.parametrize("n", [2047, 2048, 5000])
@pytest.mark.parametrize("ncrit", [1, 15, 16, 17, 32, 33, 200])
@pytest.mark.parametrize("variant", [tcb.VARIANT_TOP, tcb.VARIANT_JERKS])
def test_rows_of_every_width(n, ncrit, variant):
    x, y, z, vx, vy, vz, m = _cluster(n, 5 + ncrit)
    flags = np.random.default_rng(n).choice(np.array([1, 2, 3, 3, 3], dtype=np.uint8), size=n)
    o = oracle.evaluate(x, y, z, m, vx, vy, vz, p=4, theta=0.4, ncrit=ncrit, variant=variant, flags=flags)
    g = tcb.Gravity(p=4, ncrit=ncrit, theta=0.4, variant=variant, direct_below=0)
    out = g.evaluate(x, y, z, m, vx, vy, vz, flags=flags)
    assert g.stats()["n_p2p"] == o["stats"]["n_p2p"]
    g.close()
    sink = (flags & 1) == 1
    _close(out, o, ACC, sink)
    _close(out, o, ("pot",), sink)
    if variant == tcb.VARIANT_JERKS:
        _close(out, o, JERK, sink)


@pytest.mark.parametrize("n,ncrit", [(300, 16), (2048, 17), (9001, 64)])
@pytest.mark.parametrize("dt_param", [0.025, -0.025])
def test_time_steps_of_every_width(n, ncrit, dt_param):
    x, y, z, vx, vy, vz, m = _cluster(n, 11)
    m[5] = 0.0
    g = tcb.Gravity(p=4, ncrit=ncrit, theta=0.4, variant=tcb.VARIANT_TOP)
    out = g.evaluate_steps(x, y, z, m, vx, vy, vz, dt_param)
    g.close()
    o = oracle.evaluate_steps(x, y, z, m, vx, vy, vz, p=4, theta=0.4, ncrit=ncrit, dt_param=dt_param)
    _close(out, o, ACC)
    _close(out, o, ("timestep",))


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 127, 128, 129, 511, 513, 1040])
@pytest.mark.parametrize("jerk", [False, True])
def test_direct_sums_at_tile_edges(n, jerk):
    import torch
    b = [np.array(a) for a in ics.plummer(n, 3)]
    if n > 2:
        for q in range(3):
            b[q][1] = b[q][0]  # a coincident pair
    flags = np.random.default_rng(n).integers(0, 4, size=n).astype(np.uint8)
    src = (flags & 2) != 0
    t = [torch.tensor(a, device="cuda") for a in b]
    out = tcb.evaluate_direct_noalloc(t[0], t[1], t[2], t[6], *(t[3:6] if jerk else [None] * 3),
                                      flags=torch.tensor(flags, device="cuda"))
    torch.cuda.synchronize()
    out = {k: v.cpu().numpy() for k, v in out.items()}
    sink = (flags & 1) != 0
    o = oracle.direct(b[0], b[1], b[2], np.where(src, b[6], 0.0), *b[3:6], targets=np.arange(n, dtype=np.int32))
    for k in out:
        assert np.all(out[k][~sink] == 0)
    if src.sum() > 1 and sink.any():
        _close(out, o, ACC, sink)
        if jerk:
            _close(out, o, JERK, sink)


def test_direct_sum_in_place():
    # outputs in the inputs' own memory: the sums are those of separate outputs
    import torch
    b = [torch.tensor(a, device="cuda") for a in ics.plummer(700, 4)]
    g = tcb.Gravity(p=8, variant=tcb.VARIANT_JERKS)
    ref = g.evaluate(b[0], b[1], b[2], b[6], *b[3:6])
    out = dict(zip(ACC + JERK + ("pot",), b))
    g.evaluate(b[0], b[1], b[2], b[6], *b[3:6], out=out)
    for k in ref:
        assert torch.equal(ref[k], out[k])
    g.close()


def test_infinite_velocity_of_a_body_without_mass_in_the_sum():
    # a body that is no source leaves every other body's jerk finite, whatever its velocity
    x, y, z, vx, vy, vz, m = ics.plummer(3000, 9)
    flags = np.full(3000, 3, dtype=np.uint8)
    flags[7], vx[7] = 0, np.inf
    g = tcb.Gravity(p=4, ncrit=32, variant=tcb.VARIANT_JERKS, direct_below=1 << 20)
    out = g.evaluate(x, y, z, m, vx, vy, vz, flags=flags)
    g.close()
    assert all(np.isfinite(out[k]).all() for k in out)


@pytest.mark.parametrize("variant,p,n", [(tcb.VARIANT_JERKS, p, 98304) for p in (4, 6, 8, 10, 12, 16)] +
                         [(tcb.VARIANT_JERKS, 8, 98303), (tcb.VARIANT_TOP, 6, 98304)])
def test_far_field_of_every_order(variant, p, n):
    # the far field's form of large systems from 98,304 bodies on, and just below
    x, y, z, vx, vy, vz, m = ics.plummer(n, 21)
    flags = np.full(n, 3, dtype=np.uint8)
    flags[: n // 3] = 2
    g = tcb.Gravity(p=p, ncrit=256, theta=0.9, variant=variant, direct_below=0)
    out = g.evaluate(x, y, z, m, vx, vy, vz, flags=flags)
    o = oracle.evaluate(x, y, z, m, vx, vy, vz, p=p, theta=0.9, ncrit=256, variant=variant, flags=flags)
    assert g.stats()["n_m2l"] == o["stats"]["n_m2l"] > 0
    g.close()
    sink = (flags & 1) == 1
    _close(out, o, ACC, sink)
    _close(out, o, ("pot",), sink)
    if variant == tcb.VARIANT_JERKS:
        _close(out, o, JERK, sink)
