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


KEYS = ("x", "y", "z", "vx", "vy", "vz", "m")
OUTS = ("ax", "ay", "az", "pot", "jx", "jy", "jz")


def _device(n, seed):
    import torch
    return {k: torch.tensor(a, device="cuda") for k, a in zip(KEYS, ics.plummer_kroupa(n, seed))}


def _replay(g, d, out):
    import torch
    g.evaluate(*(d[k] for k in ("x", "y", "z", "m", "vx", "vy", "vz")), out=out)
    torch.cuda.synchronize()


def _same(a, b, what):
    import torch
    for k in OUTS:
        assert torch.equal(a[k], b[k]), (k, what)


@pytest.mark.parametrize("selector", [0, 1])
@pytest.mark.parametrize("prec", [tcb.PREC_FP64, tcb.PREC_MIXED])
def test_graph_of_a_large_system(prec, selector):
    # replays on moved bodies against the same evaluations launched directly, bit for bit
    import torch
    n = 131072
    d = _device(n, 41)
    kw = dict(p=12, ncrit=64, theta=0.4, variant=tcb.VARIANT_JERKS, precision=prec, selector=selector,
              selector_tol=3e-9)
    g, gd = tcb.Gravity(**kw), tcb.Gravity(**kw)
    g.set_graph(True)
    out, ref = ({k: torch.empty(n, dtype=torch.float64, device="cuda") for k in OUTS} for _ in range(2))
    for step in range(4):
        for k in "xyz":
            d[k] += 1e-3 * step * d["v" + k]
        _replay(g, d, out)
        assert g.graph_ready(), g.graph_note()
        _replay(gd, d, ref)
        _same(out, ref, step)
        assert g.stats()["n_m2l"] == gd.stats()["n_m2l"]
    if selector:
        assert g.stats()["class_pairs"] == gd.stats()["class_pairs"] and len(g.stats()["class_pairs"]) > 1
    g.close()
    gd.close()


@pytest.mark.parametrize("selector", [0, 1])
def test_graph_of_a_large_system_that_outgrows_its_plan(selector):
    # planned on a uniform cube, replayed on a cluster: more cells than planned.  That replay finds every list
    # empty, the call is redone and planned anew, and the |a| that order selection reads is not that replay's.
    import torch
    n = 131072
    r = np.random.default_rng(42)
    d = _device(n, 42)
    cluster = {k: d[k].clone() for k in "xyz"}
    for k in "xyz":
        d[k].copy_(torch.tensor(r.uniform(-1.0, 1.0, n), device="cuda"))
    kw = dict(p=12, ncrit=64, theta=0.5, variant=tcb.VARIANT_JERKS, selector=selector, selector_tol=3e-9)
    g, gd = tcb.Gravity(**kw), tcb.Gravity(**kw)
    g.set_graph(True)
    out, ref = ({k: torch.empty(n, dtype=torch.float64, device="cuda") for k in OUTS} for _ in range(2))
    cells = 0
    for step in range(6):
        if step == 3:
            for k in "xyz":
                d[k].copy_(cluster[k])
        _replay(g, d, out)
        assert g.graph_ready(), g.graph_note()
        _replay(gd, d, ref)
        _same(out, ref, step)
        assert step != 3 or gd.stats()["n_cells"] > 1.25 * cells + 1024
        cells = gd.stats()["n_cells"]
    g.close()
    gd.close()


@pytest.mark.parametrize("variant", [tcb.VARIANT_JERKS, tcb.VARIANT_TOP])
def test_order_classes_in_both_forms(variant):
    # 98,304 bodies, the last a massless twin of another at its place (a pair at r = 0 is left out), take the form
    # of large systems; without the twin they take the other.  The twin stands in a leaf of 57 to 62 bodies, where
    # one more changes neither the tree nor, up to some size of the cells around it, which pairs are summed
    # directly (at most 512 interactions): the first such leaf with the same lists is taken.
    n = 98304
    b = list(ics.plummer_kroupa(n - 1, 43))
    g = tcb.Gravity(p=12, ncrit=64, theta=0.4, variant=variant, selector=1, selector_tol=3e-9)

    def run(q):
        x, y, z, vx, vy, vz, m = q
        g.set_selector(0, 3e-9)
        g.evaluate(x, y, z, m, vx, vy, vz)
        g.set_selector(1, 3e-9)
        g.evaluate(x, y, z, m, vx, vy, vz)  # leaves |a| behind
        out = g.evaluate(x, y, z, m, vx, vy, vz)
        st = g.stats()
        return out, [st[k] for k in ("n_cells", "n_m2l", "n_p2p", "class_order", "class_pairs")]

    c, sc = run(b)
    cells = g.cells()
    leaves = np.nonzero((cells["nchild"] == 0) & (cells["nbody"] >= 57) & (cells["nbody"] <= 62))[0]
    for leaf in leaves[:20]:
        i = cells["perm"][cells["begin"][leaf]]
        a, sa = run([np.append(q, q[i]) for q in b[:6]] + [np.append(b[6], 0.0)])
        if sa == sc:
            break
    g.close()
    assert sa == sc and len(sa[4]) > 1
    for keys in (("ax", "ay", "az"), ("pot",)) + ((("jx", "jy", "jz"),) if variant == tcb.VARIANT_JERKS else ()):
        u, w = (np.stack([o[k][:n - 1] for k in keys]) for o in (a, c))
        nw = np.linalg.norm(w, axis=0)
        assert (np.linalg.norm(u - w, axis=0) / np.maximum(nw, 1e-3 * np.sqrt(np.mean(nw ** 2)))).max() < 1e-11
