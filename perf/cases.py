"""The work that users of this library have it do, as cases to be timed.

A case is one call through the public entry points (``Gravity.evaluate``, ``evaluate_steps``,
``step_leapfrog``, ``evolve_hold_dkd``) on a star cluster made from a seed: direct sums of small
groups, the evaluations and time-step passes that a block-time-step integrator asks for, single
evaluations of clusters from ten thousand to a million bodies in both precisions, and the
shared-step leapfrog of a four-million-body cluster.  Inputs are made on the GPU in Henon units.
"""
import math

import numpy as np
import torch

import taichi_collisional_b200 as tcb

TREE = {"top": tcb.VARIANT_TOP, "jerks": tcb.VARIANT_JERKS}
PREC = {"fp64": tcb.PREC_FP64, "mixed": tcb.PREC_MIXED}
VEL = ("vx", "vy", "vz")

DEFAULTS = {"ics": "plummer_kroupa", "tree": "jerks", "precision": "fp64", "p": 12, "ncrit": 64, "theta": 0.4,
            "mac": "theta", "selector": 0, "memory": "device", "sinks": "all"}


def case(name, kind, n, **kw):
    c = dict(DEFAULTS, kind=kind, n=n, **kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # A small group in the jerks tree: below 8,000 bodies the call is a direct sum.
        case("direct_500", "evaluate", 500),
        # The largest such group but for the last bodies, a ragged size.
        case("direct_7001", "evaluate", 7001),
        # The time-step pass of the block-time-step integrator on one of its middle levels.
        case("steps_2000", "steps", 2000, tree="top", p=8),
        # One kick of that integrator: sources kick sinks (the fast third of a system), lists by the
        # error-controlled criterion.
        case("kick_12345_error_mac", "evaluate", 12345, tree="top", p=8, mac="error", sinks="third"),
        # The small plain run: equal masses, theta criterion, a host program's own arrays.
        case("plummer_16k_host", "evaluate", 16384, ics="plummer", tree="top", p=8, theta=0.5, memory="host"),
        # A whole step of the block-time-step integrator on a small cluster.
        case("evolve_1024", "evolve", 1024, tree="top", p=8, mac="error"),
        # The jerks tree as the original program calls it: its error-controlled criterion.
        case("jerks_65537_error_mac", "evaluate", 65537, p=10, mac="error"),
        # A cluster evaluated in FP64 with jerks, the parity form.
        case("jerks_131k_fp64", "evaluate", 131072),
        # A million equal-mass bodies at order 10 with the FP32 near field.
        case("plummer_1m_mixed_p10", "evaluate", 1048576, ics="plummer", precision="mixed", p=10),
        # A deep, uneven tree (a fractal cluster) with small leaves and per-pair orders.
        case("fractal_500k_orders", "evaluate", 500000, ics="fractal", precision="mixed", ncrit=32, selector=1),
        # The accurate far field: order 16 in FP64.
        case("jerks_750k_p16", "evaluate", 750001, p=16, theta=0.5),
        # The production step: leapfrog of four million bodies, mixed precision, learned per-pair
        # orders, replayed as one CUDA graph.
        case("leapfrog_4m_learned", "leapfrog", 4194304, precision="mixed", selector=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["direct", "steps", "kick", "evaluate", "evaluate", "evaluate", "leapfrog", "evolve"])
    ics = rng.choice(["plummer_kroupa", "plummer_kroupa", "plummer", "fractal"])
    if kind == "direct":
        return case(None, "evaluate", _log_int(rng, 64, 7999), ics=ics)
    if kind == "steps":
        return case(None, "steps", _log_int(rng, 300, 100000), ics=ics, tree="top", p=8)
    if kind == "kick":
        return case(None, "evaluate", _log_int(rng, 300, 100000), ics=ics, tree="top", p=8, mac="error",
                    sinks=rng.choice(["all", "third", "half"]))
    if kind == "evolve":
        return case(None, "evolve", _log_int(rng, 200, 1024), tree="top", p=8, mac="error")
    if kind == "leapfrog":
        return case(None, "leapfrog", _log_int(rng, 50000, 2000000), precision="mixed", p=12,
                    ncrit=rng.choice([32, 64]), selector=rng.choice([0, 1, 2]))
    p = rng.choice([6, 8, 10, 12, 16])
    mac = rng.choice(["theta", "theta", "theta", "error"])
    return case(None, "evaluate", _log_int(rng, 9000, 200000 if mac == "error" else 1000000), ics=ics, p=p,
                tree=rng.choice(["top", "jerks"]), precision=rng.choice(["fp64", "mixed"]), mac=mac,
                theta=rng.choice([0.4, 0.5]), ncrit=rng.choice([32, 64, 128]),
                memory=rng.choice(["device", "device", "host"]))


# ---- initial conditions on the GPU: the distributions of taichi_collisional_b200.ics ----
def _unit(n, g):
    ct = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    ph = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
    st = torch.sqrt(1 - ct * ct)
    return torch.stack([st * torch.cos(ph), st * torch.sin(ph), ct], 1)


def _plummer(n, g):
    """Plummer sphere inside r < 10 (Aarseth, Henon & Wielen 1974): positions and velocities, n x 3."""
    a, rmax = tcb.ics.PLUMMER_SCALE, 10.0
    top = (1 + (a / rmax) ** 2) ** -1.5  # the mass inside rmax
    x = (1e-10 + (1 - 1e-10) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)) * top
    r = 1 / torch.sqrt(x ** (-2.0 / 3.0) - 1)
    q = torch.empty_like(r)
    todo = torch.arange(n, device="cuda")
    while len(todo):  # speed by rejection on q^2 (1 - q^2)^3.5
        t = torch.rand(2, len(todo), generator=g, device="cuda", dtype=torch.float64)
        ok = t[1] * 0.1 < t[0] ** 2 * (1 - t[0] ** 2) ** 3.5
        q[todo[ok]] = t[0][ok]
        todo = todo[~ok]
    v = q * math.sqrt(2.0) * (1 + r * r) ** -0.25
    return _unit(n, g) * (r * a)[:, None], _unit(n, g) * (v / math.sqrt(a))[:, None]


def _kroupa(n, g):
    """Kroupa (2001) masses between 0.08 and 100 solar masses, summing to 1."""
    u = torch.rand(2, n, generator=g, device="cuda", dtype=torch.float64)

    def integral(s, lo, hi):
        return (hi ** (1 - s) - lo ** (1 - s)) / (1 - s)

    def inverse(s, lo, hi, t):
        return (lo ** (1 - s) + t * (hi ** (1 - s) - lo ** (1 - s))) ** (1 / (1 - s))

    low, high = integral(1.3, 0.08, 0.5), 0.5 * integral(2.3, 0.5, 100.0)
    m = torch.where(u[0] < low / (low + high), inverse(1.3, 0.08, 0.5, u[1]), inverse(2.3, 0.5, 100.0, u[1]))
    return m / m.sum()


def _fractal(n, g):
    """Box fractal of dimension 1.6 (Goodwin & Whitworth 2004), cold, virial ratio about 0.3."""
    f64 = dict(device="cuda", dtype=torch.float64)
    surv, half = 2.0 ** (1.6 - 3.0), 1.0
    offs = torch.tensor([[(i >> d & 1) * 2.0 - 1.0 for d in range(3)] for i in range(8)], **f64)
    c, v = torch.zeros(1, 3, **f64), torch.zeros(1, 3, **f64)
    while len(c) * surv * 8 < 4 * n or len(c) < n:
        half *= 0.5
        k = (c[:, None, :] + offs[None] * half).reshape(-1, 3)
        kv = v.repeat_interleave(8, 0) + half * torch.randn(len(k), 3, generator=g, **f64)
        keep = torch.rand(len(k), generator=g, **f64) < surv
        if len(k) <= 4096:
            keep[torch.randint(len(k), (1,), generator=g, device="cuda")] = True  # the cluster does not die out
        k, v = k[keep], kv[keep]
        c = k + 0.1 * half * (torch.rand(k.shape, generator=g, **f64) * 2 - 1)
    pick = torch.randperm(len(c), generator=g, device="cuda")[:n]
    x = c[pick] + half * (torch.rand(n, 3, generator=g, **f64) * 2 - 1)
    v = v[pick] + half * torch.randn(n, 3, generator=g, **f64)
    x, v = x - x.mean(0), v - v.mean(0)
    s = torch.randint(n, (256,), generator=g, device="cuda")
    phi = sum(torch.nan_to_num(1 / torch.cdist(x[s], b), posinf=0.0).sum(1) for b in x.split(1 << 16)) / n
    w = 0.5 * float(phi.mean())  # minus the potential energy
    v = v * math.sqrt(0.3 * w / float(0.5 * (v * v).sum() / n))
    scale = 0.7 * w / 0.25  # to a total energy of -1/4
    return x * scale, v / math.sqrt(scale)


def _bodies(c, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = c["n"]
    x, v = _fractal(n, g) if c["ics"] == "fractal" else _plummer(n, g)
    m = _kroupa(n, g) if c["ics"] == "plummer_kroupa" else torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    x = x - (m[:, None] * x).sum(0)
    v = v - (m[:, None] * v).sum(0)
    b = {k: x[:, i].contiguous() for i, k in enumerate("xyz")}
    b.update({k: v[:, i].contiguous() for i, k in enumerate(VEL)})
    b["m"] = m
    b["flags"] = None
    if c["sinks"] != "all":  # bit 0: sink, bit 1: source; the first bodies are kicked by the others
        b["flags"] = torch.full((n,), 2, device="cuda", dtype=torch.uint8)
        b["flags"][: n // (3 if c["sinks"] == "third" else 2)] = 1
    return b


def prepare(c, seed):
    b = _bodies(c, seed)
    g = tcb.Gravity(p=c["p"], ncrit=c["ncrit"], theta=c["theta"], variant=TREE[c["tree"]],
                    precision=PREC[c["precision"]])
    if c["mac"] == "error":
        g.set_error_mac(True, 2e-7 if c["tree"] == "top" else 2e-8)
    s = {"case": c, "g": g, "b": b}
    if c["selector"] == 2:  # trained once on the program's own bodies
        g.train_selector(*(b[k] for k in ("x", "y", "z", "m") + VEL), nsamples=16384, iters=1500, seed=5)
    if c["selector"]:
        g.set_selector(c["selector"], 3e-9)
    if c["kind"] == "leapfrog" or c["selector"]:  # a stepping program has evaluated the state before
        s["out"] = _evaluate(g, b, c)
    if c["kind"] == "leapfrog":
        g.set_graph(True)
    if c["kind"] == "evolve":
        for k in ("ex", "ey", "ez", "timestep", "pot"):
            b[k] = torch.zeros_like(b["x"])
        b["id"] = torch.arange(c["n"], dtype=torch.int32, device="cuda")
        b.pop("flags")
    if c["memory"] == "host":
        s["b"] = {k: None if t is None else t.cpu().numpy() for k, t in b.items()}
    return s


def _evaluate(g, b, c):
    v = [b[k] for k in VEL] if c["tree"] == "jerks" else [None] * 3
    return g.evaluate(b["x"], b["y"], b["z"], b["m"], *v, flags=b["flags"])


def run(s):
    c, g, b = s["case"], s["g"], s["b"]
    if c["kind"] == "steps":
        return g.evaluate_steps(b["x"], b["y"], b["z"], b["m"], *(b[k] for k in VEL), dt_param=0.025)
    if c["kind"] == "leapfrog":
        g.step_leapfrog(b, s["out"], LEAPFROG_DT)
        return dict(s["out"], **{k: b[k] for k in ("x", "y", "z") + VEL})
    if c["kind"] == "evolve":
        g.evolve_hold_dkd(b, 0.025, EVOLVE_DT)
        return b
    return _evaluate(g, b, c)


LEAPFROG_DT = 1.0 / 4096
EVOLVE_DT = 1.0 / 64


def work(c):
    """Inputs and outputs once; the pair sums and far-field translations that the tree leaves, about
    60 ncrit near-field partners and 36 (64 / ncrit) far cells a body at theta = 0.4, and 5 (p + 1)^3
    operations for each translated expansion (the jerks tree has two)."""
    n, jerk = c["n"], c["tree"] == "jerks"
    pair = 45.0 if jerk or c["kind"] == "steps" else 22.0
    nbytes = 8.0 * n * ((7 + 7) if jerk else (4 + 4)) + (56.0 * n if c["kind"] in ("steps", "leapfrog") else 0)
    if n < (8000 if jerk else c["ncrit"]) and c["kind"] != "steps":
        return {"bytes": nbytes, "flops": pair * n * n}
    open3 = (0.4 / c["theta"]) ** 3
    near = n * min(float(n), 60.0 * c["ncrit"] * open3)
    far = 36.0 * (64.0 / c["ncrit"]) * n * open3 * 5 * (c["p"] + 1) ** 3 * (2 if jerk else 1)
    if n < 1000 * c["ncrit"]:  # shallow trees: fewer far cells
        far *= n / (1000.0 * c["ncrit"])
    if c["selector"]:
        far *= 0.55
    if c["kind"] == "steps":
        far = 0.0
    once = {"bytes": nbytes, "flops": pair * near + far}
    if c["kind"] == "evolve":  # some hundreds of evaluations on ever smaller systems: about 30 whole ones
        return {"bytes": 30 * nbytes, "flops": 30 * once["flops"]}
    return once


def _direct(b, jerk):
    """Accelerations, potential and jerks by direct summation in 64 bits, plain torch on the GPU."""
    n = len(b["x"])
    src = torch.ones(n, dtype=torch.bool, device="cuda") if b["flags"] is None else (b["flags"] & 2) != 0
    sink = torch.ones_like(src) if b["flags"] is None else (b["flags"] & 1) != 0
    X, V, m = [b[k][src] for k in "xyz"], [b[k][src] for k in VEL], b["m"][src]
    out = {k: torch.zeros(n, dtype=torch.float64, device="cuda")
           for k in ("ax", "ay", "az", "pot") + (("jx", "jy", "jz") if jerk else ())}
    for at in torch.nonzero(sink)[:, 0].split(max(1, (1 << 25) // n)):
        d = [X[i][None] - b[k][at][:, None] for i, k in enumerate("xyz")]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        inv2 = torch.where(r2 > 0, 1 / r2, torch.zeros_like(r2))
        f = m[None] * torch.sqrt(inv2)
        out["pot"][at] = f.sum(1)
        f *= inv2
        for i, k in enumerate(("ax", "ay", "az")):
            out[k][at] = (d[i] * f).sum(1)
        if jerk:
            w = [V[i][None] - b[k][at][:, None] for i, k in enumerate(VEL)]
            h = (d[0] * w[0] + d[1] * w[1] + d[2] * w[2]) * inv2 * f * 3
            for i, k in enumerate(("jx", "jy", "jz")):
                out[k][at] = (w[i] * f - d[i] * h).sum(1)
    return out


def exact(c, seed):
    # 64-bit direct sums; the time-step pass (near field of its own tree) and the hierarchical step
    # have no such value, and over 300,000 bodies the sums take too long
    if c["kind"] in ("steps", "evolve") or c["n"] > 300000:
        return None
    b, jerk = _bodies(c, seed), c["tree"] == "jerks"
    if c["kind"] == "leapfrog":
        dt = LEAPFROG_DT
        a = _direct(b, False)
        for k, w, q in zip("xyz", VEL, ("ax", "ay", "az")):
            b[w] = b[w] + a[q] * (0.5 * dt)
            b[k] = b[k] + b[w] * dt
        o = _direct(b, True)
        return dict(o, **{k: b[k] for k in "xyz"},
                    **{w: b[w] + o[q] * (0.5 * dt) for w, q in zip(VEL, ("ax", "ay", "az"))})
    o = _direct(b, jerk)
    return {k: t.cpu().numpy() for k, t in o.items()} if c["memory"] == "host" else o
