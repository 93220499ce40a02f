"""Interaction lists of trees with more cells than the list bitmaps cover, and what planning a graph holds.

Tolerance: an accepted pair's expansion of order p = 4 at theta = 0.5 is cut at theta^(p + 1), 0.03 of the
pair's own field; the pairs' errors point every way and the near field has none, so the rms error over a
body's field stays well under a third of that, 1e-2.  A target that loses pairs is off by about its field."""
import numpy as np
import pytest

import taichi_collisional_b200 as tcb
from taichi_collisional_b200 import ics

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BITMAP_CELLS = 416 << 10  # kListMaxCells
KEYS = ("x", "y", "z", "vx", "vy", "vz", "m")


def _many_cells(seed):
    """A cluster whose tree of single-body leaves has about two million cells (keys of 42 bits)."""
    return {k: torch.tensor(np.ascontiguousarray(a), device="cuda") for k, a in zip(KEYS, ics.plummer(1250000, seed))}


def _gravity(**kw):
    return tcb.Gravity(p=4, ncrit=1, theta=0.5, variant=tcb.VARIANT_JERKS, direct_below=0, **kw)


def _outs(n):
    return {k: torch.empty(n, dtype=torch.float64, device="cuda") for k in ("ax", "ay", "az", "pot", "jx", "jy", "jz")}


def _evaluate(g, d, out=None):
    return g.evaluate(*(d[k] for k in ("x", "y", "z", "m", "vx", "vy", "vz")), out=out)


def test_forces_of_a_tree_beyond_the_list_bitmaps():
    d = _many_cells(31)
    idx = np.random.default_rng(31).choice(len(d["x"]), 512, replace=False)
    g = _gravity()
    out = _evaluate(g, d)
    assert max(BITMAP_CELLS, 1 << 20) < g.stats()["n_cells"] < 1 << 21
    ref = g.direct_sums(*(d[k] for k in ("x", "y", "z", "m")), idx)
    g.close()
    for keys in (("ax", "ay", "az"), ("pot",)):
        a = np.stack([out[k].cpu().numpy()[idx] for k in keys])
        b = np.stack([ref[k] for k in keys])
        err = np.sqrt(np.mean(np.sum((a - b) ** 2, 0)) / np.mean(np.sum(b ** 2, 0)))
        assert err < 1e-2, (keys, err)


def test_graph_of_a_tree_beyond_the_list_bitmaps():
    # captured and replayed like any other; replays take no memory
    d = _many_cells(32)
    n = len(d["x"])
    g, gd = _gravity(), _gravity()
    g.set_graph(True)
    out, ref = _outs(n), _outs(n)
    for step in range(3):
        for k in "xyz":
            d[k] += 1e-4 * step * d["v" + k]
        _evaluate(g, d, out)
        assert g.graph_ready(), g.graph_note()
        _evaluate(gd, d, ref)
        torch.cuda.synchronize()
        assert g.stats()["n_cells"] == gd.stats()["n_cells"] > BITMAP_CELLS
        for k in ref:
            assert torch.equal(out[k], ref[k]), (k, step)
        free = torch.cuda.mem_get_info()[0]
        assert step == 0 or free == last, step
        last = free
    g.close()
    gd.close()


def test_planning_again_takes_no_more_memory():
    # other output buffers: a new plan each call, of the same capacities
    d = {k: torch.tensor(np.ascontiguousarray(a), device="cuda") for k, a in zip(KEYS, ics.plummer(65536, 33))}
    g = tcb.Gravity(p=4, ncrit=64, theta=0.5, variant=tcb.VARIANT_JERKS)
    g.set_graph(True)
    outs = [_outs(65536) for _ in range(2)]
    free = []
    for k in range(10):
        _evaluate(g, d, outs[k % 2])
        assert g.graph_ready(), g.graph_note()
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])
    g.close()
    assert len(set(free[2:])) == 1, free


@pytest.mark.parametrize("graph", [False, True])
def test_a_context_grows_with_its_system(graph):
    # a frontier sized for a small system overflows on a large one; the call grows it and answers as a
    # context that never saw the small one
    def run(g, n):
        d = {k: torch.tensor(np.ascontiguousarray(a), device="cuda") for k, a in zip(KEYS, ics.plummer(n, 34))}
        out = _evaluate(g, d)
        torch.cuda.synchronize()
        return out, g.stats()

    kw = dict(p=4, ncrit=64, theta=0.5, variant=tcb.VARIANT_JERKS, direct_below=0)
    g, fresh = tcb.Gravity(**kw), tcb.Gravity(**kw)
    g.set_graph(graph)
    run(g, 300)
    out, st = run(g, 600000)
    ref, sr = run(fresh, 600000)
    assert (st["n_cells"], st["n_m2l"], st["n_p2p"]) == (sr["n_cells"], sr["n_m2l"], sr["n_p2p"])
    for k in ref:
        assert torch.equal(out[k], ref[k]), k
    g.close()
    fresh.close()


@pytest.mark.parametrize("variant,ncrit", [(tcb.VARIANT_JERKS, 4), (tcb.VARIANT_JERKS, 8), (tcb.VARIANT_TOP, 8)])
def test_a_tree_of_more_cells_than_the_first_estimate(variant, ncrit):
    # Small leaves: more than the n / 4 (or 2 n / ncrit) cells that the buffers first hold.  Sums of at most
    # n = 9,000 FP64 terms in another order than the oracle's: (n + 10) 2^-53 = 1e-12 of the terms' magnitudes,
    # of which the field is a tenth; twice that.
    import oracle
    n = 9000
    x, y, z, vx, vy, vz, m = ics.plummer(n, 35)
    o = oracle.evaluate(x, y, z, m, vx, vy, vz, p=4, theta=0.5, ncrit=ncrit, variant=variant)
    g = tcb.Gravity(p=4, ncrit=ncrit, theta=0.5, variant=variant, direct_below=0)
    for _ in range(2):
        out = g.evaluate(x, y, z, m, vx, vy, vz)
        assert g.stats()["n_cells"] > 2 * n // min(ncrit, 8) + 1024
        a, b = (np.stack([q[k] for k in ("ax", "ay", "az")]) for q in (out, o))
        nb = np.linalg.norm(b, axis=0)
        assert (np.linalg.norm(a - b, axis=0) / np.maximum(nb, 1e-3 * np.sqrt(np.mean(nb ** 2)))).max() < 2e-11
    g.close()


def test_a_replay_that_outgrows_the_list_bitmaps():
    # planned on a tree just below the bitmaps' limit, replayed on one above it: the call is redone, planned
    # anew with sorted lists, and the next call replays that
    n = 280000
    r = np.random.default_rng(36)
    d = {k: torch.tensor(np.ascontiguousarray(a), device="cuda") for k, a in zip(KEYS, ics.plummer(n, 36))}
    for k in "xyz":
        d[k].copy_(torch.tensor(r.uniform(-1.0, 1.0, n), device="cuda"))
    g, gd = _gravity(), _gravity()
    g.set_graph(True)
    out, ref = _outs(n), _outs(n)
    for step in range(4):
        if step == 2:  # close pairs: chains of cells down to each
            for k in "xyz":
                d[k][:14000] = d[k][14000:28000] + torch.tensor(1e-3 * r.standard_normal(14000), device="cuda")
        _evaluate(g, d, out)
        assert g.graph_ready(), g.graph_note()
        _evaluate(gd, d, ref)
        torch.cuda.synchronize()
        cells = g.stats()["n_cells"]
        assert cells == gd.stats()["n_cells"] and (cells > BITMAP_CELLS) == (step >= 2) and cells > 350000
        for k in ref:
            assert torch.equal(out[k], ref[k]), (k, step)
    g.close()
    gd.close()
