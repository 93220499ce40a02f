"""The far field's two forms at the rule between them, and the form of large systems in a captured graph.

Tolerance against the oracle: sums of FP64 terms in another order, as in test_gpu_rows.py: 1e-11."""
import numpy as np
import pytest

import oracle
import taichi_collisional_b200 as tcb
from taichi_collisional_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,p,ncrit", [(tcb.VARIANT_JERKS, p, 128) for p in (4, 6, 8, 10)] +
                         [(tcb.VARIANT_TOP, 6, 64), (tcb.VARIANT_TOP, 12, 128), (tcb.VARIANT_TOP, 12, 129),
                          (tcb.VARIANT_JERKS, 8, 129)])
def test_far_field_at_the_fewest_targets_of_its_form(variant, p, ncrit):
    # the work items (expansions of a target) from which the form of large systems takes over, and just below
    n = 98304
    x, y, z, vx, vy, vz, m = ics.plummer(n, 22)
    flags = np.full(n, 3, dtype=np.uint8)
    flags[: n // 3] = 2
    g = tcb.Gravity(p=p, ncrit=ncrit, theta=0.9, variant=variant, direct_below=0)
    out = g.evaluate(x, y, z, m, vx, vy, vz, flags=flags)
    o = oracle.evaluate(x, y, z, m, vx, vy, vz, p=p, theta=0.9, ncrit=ncrit, variant=variant, flags=flags)
    assert g.stats()["n_m2l"] == o["stats"]["n_m2l"] > 0
    g.close()
    sink = (flags & 1) == 1
    for keys in (("ax", "ay", "az"), ("pot",)) + ((("jx", "jy", "jz"),) if variant == tcb.VARIANT_JERKS else ()):
        a, b = (np.stack(q) for q in zip(*[(out[k][sink], o[k][sink]) for k in keys]))
        nb = np.linalg.norm(b, axis=0)
        assert (np.linalg.norm(a - b, axis=0) / np.maximum(nb, 1e-3 * np.sqrt(np.mean(nb ** 2)))).max() < 1e-11
