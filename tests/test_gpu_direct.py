"""Potentials of the direct sums at the edges of their tiles (accelerations and jerks: test_gpu_rows.py).

Tolerance: sums of at most n = 1,040 positive FP64 terms of a few roundings each: (n + 10) 2^-53 = 1.2e-13 of
the value."""
import numpy as np
import pytest

import oracle
import taichi_collisional_b200 as tcb
from taichi_collisional_b200 import ics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 15, 17, 127, 128, 129, 511, 513, 1040])
@pytest.mark.parametrize("jerk", [False, True])
def test_potential_at_tile_edges(n, jerk):
    import torch
    b = [np.array(a) for a in ics.plummer(n, 3)]
    flags = np.random.default_rng(n).integers(0, 4, size=n).astype(np.uint8)
    t = [torch.tensor(a, device="cuda") for a in b]
    out = tcb.evaluate_direct_noalloc(t[0], t[1], t[2], t[6], *(t[3:6] if jerk else [None] * 3),
                                      flags=torch.tensor(flags, device="cuda"))
    torch.cuda.synchronize()
    sink = (flags & 1) != 0
    o = oracle.direct(b[0], b[1], b[2], np.where((flags & 2) != 0, b[6], 0.0), *b[3:6])
    np.testing.assert_allclose(out["pot"].cpu().numpy()[sink], o["pot"][sink], rtol=1.2e-13)
