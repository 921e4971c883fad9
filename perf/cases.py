"""Performance cases: what users of this framework have it do, through its public calls.

A case names an operation (generate, batch, vjp, inverse, host), a process of
gpu_phs_gb300.processes, a number of events and the options in use (precision, beams).
``prepare`` makes what a program holds before the call, ``run`` is the call, ``exact`` the
same map restated in plain torch float64.
"""
import math

import numpy as np
import torch

from gpu_phs_gb300 import processes as P
from gpu_phs_gb300.api import PRECISION_F32X2, PRECISION_F64, Batch, Events, PhaseSpace

DEV = "cuda"
CHUNK = 1 << 20   # events of one piece of the restatement below (bounds its memory)


def listed():
    return [
        # a generator called event loop by event loop: a thousand e+e- -> WW events per call,
        # where launches and latency count
        _case("ww_small", "generate", "ww", 1000),
        # the headline configuration: tt -> 6f, 1e7 events per call, FP64
        _case("tt_f64", "generate", "tt", 10_000_000),
        # the same tree in FP32 pairs, a ragged number of events
        _case("tt_f32x2", "generate", "tt", 1_000_003, precision="f32x2"),
        # 2 -> 6 massless partons at 13 TeV: most events fail the kinematic test
        _case("pp6j_f64", "generate", "precision", 3_000_001),
        _case("pp6j_f32x2", "generate", "precision", 1 << 24, precision="f32x2"),
        # 64 channel trees of 3 to 8 particles with uneven event counts in one launch
        _case("batch64_f64", "batch", "batched", 1 << 22, n_channels=64, tree_seed=2024),
        _case("batch64_f32x2", "batch", "batched", 1 << 24, n_channels=64, tree_seed=2024,
              precision="f32x2"),
        # hadron-collider mode: every event has its own beam energies
        _case("tt_beams_f64", "generate", "tt", 500_000, beams="event"),
        # the largest trees the API takes: three channels over 12 particles
        _case("nested12_f64", "generate", "nested", 300_001, n_out=12),
        # gradients of momenta and Jacobians (training an integrator, fitting masses)
        _case("tt_vjp", "vjp", "tt", 1_000_000),
        # multi-channel weights: every event inverted in all 16 channels of a process
        _case("inverse16", "inverse", "random", 200_000, n_out=6, n_channels=16, tree_seed=5),
        # a host program's call: pinned host arrays in and out
        _case("tt_host", "host", "tt", 1_500_000),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["generate", "generate", "generate", "batch", "vjp", "inverse", "host"])
    precision = rng.choice(["f64", "f32x2"])
    if op == "batch":
        return _case(None, op, "batched", log(20_000, 1 << 22), n_channels=rng.randint(2, 80),
                     tree_seed=rng.randrange(1 << 20), precision=precision)
    if op == "inverse":
        return _case(None, op, "random", log(1000, 150_000), n_out=rng.randint(4, 7),
                     n_channels=rng.randint(2, 16), tree_seed=rng.randrange(1 << 20),
                     beams=rng.choice(["equal", "lab"]))
    if op == "vjp":
        return _case(None, op, rng.choice(["ww", "tt"]), log(1000, 1_000_000),
                     beams=rng.choice(["equal", "lab"]))
    if op == "host":
        return _case(None, op, rng.choice(["ww", "tt"]), log(1000, 1_500_000))
    kind = rng.choice(["ww", "tt", "precision", "random", "nested"])
    n = log(1000, 200_000 if kind == "nested" else 3_000_000)
    beams = rng.choice(["equal", "equal", "lab", "event"])
    if kind == "random":
        return _case(None, op, kind, n, n_out=rng.randint(3, 8), n_channels=rng.randint(1, 12),
                     tree_seed=rng.randrange(1 << 20), precision=precision, beams=beams)
    return _case(None, op, kind, n, n_out=rng.randint(8, 12) if kind == "nested" else 0,
                 precision=precision, beams=beams)


def _case(name, op, process, events, n_out=0, n_channels=1, tree_seed=0, precision="f64",
          beams="equal"):
    c = {"op": op, "process": process, "events": int(events), "n_out": n_out,
         "n_channels": n_channels, "tree_seed": tree_seed, "precision": precision, "beams": beams}
    return dict(c, name=name) if name else c


# ------------------------------------------------------------------ what a program holds
def _processes(case):
    """The processes of a case and the events of each channel."""
    kind, n = case["process"], case["events"]
    if kind == "batched":
        procs, counts = P.batched(case["tree_seed"], case["n_channels"], n)
        return procs, counts
    if kind == "random":
        proc = P.random_process(np.random.default_rng(case["tree_seed"]), case["n_out"],
                                case["n_channels"])
    elif kind == "nested":
        proc = P.nested_resonances(case["n_out"])
    else:
        proc = {"ww": P.ww, "tt": P.tt, "precision": P.precision}[kind]()
    w = np.arange(1, proc.n_channels + 1, dtype=np.float64) ** -1.5
    counts = np.floor(w / w.sum() * n).astype(np.int64)
    counts[0] += n - int(counts.sum())
    return [proc], counts


def _beams(case, proc):
    """Uniform beam energies: equal, or asymmetric at the nominal sqrt(s)."""
    e = 0.5 * proc.sqrts
    return (e, e) if case["beams"] != "lab" else (1.2 * e, e / 1.2)


def _inputs(case, seed):
    """(processes, counts, x flat or [n, n_x], per-event beams or None, generator)."""
    procs, counts = _processes(case)
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    if case["op"] == "batch":
        size = int(sum(p.n_x * int(c) for p, c in zip(procs, counts)))
        x = torch.rand(size, dtype=torch.float64, device=DEV, generator=g)
    else:
        x = torch.rand((case["events"], procs[0].n_x), dtype=torch.float64, device=DEV, generator=g)
    energies = None
    if case["beams"] == "event":
        energies = tuple(procs[0].sqrts * (0.3 + 0.4 * torch.rand(
            case["events"], dtype=torch.float64, device=DEV, generator=g)) for _ in range(2))
    return procs, counts, x, energies, g


def _counts_arg(proc, counts):
    return counts if proc.n_channels > 1 else None


def prepare(case, seed):
    procs, counts, x, energies, g = _inputs(case, seed)
    op, prec = case["op"], PRECISION_F32X2 if case["precision"] == "f32x2" else PRECISION_F64
    state = {"op": op, "x": x}
    if op == "batch":
        spaces = [PhaseSpace(p, *_beams(case, p)) for p in procs]
        state.update(batch=Batch(spaces), counts=counts)
        state["batch"].set_precision(prec)
        return state
    proc = procs[0]
    ps = PhaseSpace(proc, *_beams(case, proc))
    ps.set_precision(prec)
    state.update(ps=ps, counts=_counts_arg(proc, counts), energies=energies)
    n = case["events"]
    if op == "vjp":
        state["pbar"] = torch.randn((n, proc.n_out, 4), dtype=torch.float64, device=DEV, generator=g)
        state["jbar"] = torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
    elif op == "inverse":
        # the events to invert, from the restatement: the same momenta for every version
        p, factor, _, ok = _forward(proc, counts, x, case)
        state.update(p=p, factor=factor, ok=ok)
    elif op == "host":
        state["x"] = x.cpu().pin_memory()
        state["out"] = Events(*[torch.empty(s, dtype=t).pin_memory() for s, t in (
            ((n, proc.n_out, 4), torch.float64), (n, torch.float64), (n, torch.float64),
            (n, torch.uint8))])
    return state


def run(state):
    op, x = state["op"], state["x"]
    if op == "batch":
        return state["batch"].generate(x, state["counts"])
    ps, counts = state["ps"], state["counts"]
    if op == "vjp":
        return ps.vjp(x, state["pbar"], state["jbar"], counts)
    if op == "inverse":
        return ps.inverse(state["p"], counts, ok=state["ok"], x=x, factor=state["factor"])
    if op == "host":
        ev = ps.generate_host(x, counts, out=state["out"])
    elif state["energies"] is not None:
        ev = ps.generate_beams(x, *state["energies"], counts)
    else:
        ev = ps.generate(x, counts)
    return ev.p, ev.factor, ev.volume, ev.ok


# share of the events that pass the kinematic test: only those need angles and boosts
OK_SHARE = {"ww": 0.99, "tt": 0.99, "precision": 0.04, "batched": 0.2, "random": 0.2, "nested": 0.5}


def work(case):
    """Bytes: inputs once, outputs once.  Operations: add, multiply, divide, square root and
    each elementary function one each, in the 64-bit algorithm."""
    procs, counts = _processes(case)
    share = OK_SHARE[case["process"]]
    n_bytes = flops = 0.0
    at = 0
    for proc in procs:
        own = counts[at:at + proc.n_channels]
        at += proc.n_channels
        n, visits = float(own.sum()), proc.n_out - 1
        row = 8 * proc.n_x + 32 * proc.n_out + 17
        test = (visits - 1) * 10 + visits * 9                    # mappings, Kallen and the test
        walk = visits * 24 + (visits - 1) * 70 + proc.n_out * 14   # angles, frames, momenta
        if case["op"] == "inverse":
            n_bytes += n * (row - 8 + proc.n_channels * 8 * (proc.n_x + 1))
            flops += n * share * (proc.n_channels - 1) * (test + walk)
        elif case["op"] == "vjp":
            n_bytes += n * (16 * proc.n_x + 32 * proc.n_out + 8 + 16 * (proc.n_out - 2))
            flops += n * 3 * (test + walk)
        else:
            n_bytes += n * (row + (16 if case["beams"] == "event" else 0))
            flops += n * (test + share * walk)
    return {"bytes": n_bytes, "flops": flops}


# ------------------------------------------------------------ the map in plain 64-bit torch
def exact(case, seed):
    procs, counts, x, energies, g = _inputs(case, seed)
    proc, op = procs[0], case["op"]
    if op == "batch":
        parts, at, xat = [], 0, 0
        for p, c in zip(procs, counts):
            c = int(c)
            xs = x[xat:xat + c * p.n_x].view(c, p.n_x)
            parts.append(_forward(p, np.array([c]), xs, case))
            xat += c * p.n_x
        out = [torch.cat([q[k].reshape(-1) for q in parts]) for k in range(3)]
        return out[0], out[1], out[2], None
    if op == "vjp":
        n = case["events"]
        pbar = torch.randn((n, proc.n_out, 4), dtype=torch.float64, device=DEV, generator=g)
        jbar = torch.randn(n, dtype=torch.float64, device=DEV, generator=g)
        return _gradients(proc, x, pbar, jbar, case)
    if op == "inverse":
        p, factor, _, ok = _forward(proc, counts, x, case)
        return _inverse(proc, counts, p, ok, x, factor, case)
    p, factor, volume, _ = _forward(proc, counts, x, case, energies)
    if op == "host":
        p, factor, volume = p.cpu(), factor.cpu(), volume.cpu()
    return p, factor, volume, None


class _Tree:
    """One channel: daughters, mappings, mass sums and the order in which it takes x."""

    def __init__(self, proc, c):
        self.n_out, self.root = proc.n_out, (1 << proc.n_out) - 1
        self.kids, self.map, self.leaf_m = {}, {}, {}
        self.m_min, self.x_msq, self.x_ang = {}, {}, {}
        for j in range(proc.n_out):
            self.leaf_m[1 << j] = float(proc.flv_masses[proc.n_in + j])

        def post(code):
            if not proc.has_children[c, code - 1]:
                self.m_min[code] = self.leaf_m[code]
                return
            a, b = int(proc.d1[c, code - 1]), int(proc.d2[c, code - 1])
            self.kids[code] = (a, b)
            self.map[code] = (int(proc.map_ids[c, code - 1]), float(proc.map_masses[c, code - 1]),
                              float(proc.map_widths[c, code - 1]))
            post(a)
            post(b)
            self.m_min[code] = self.m_min[a] + self.m_min[b]
            if code != self.root:
                self.x_msq[code] = len(self.x_msq)

        def pre(code):
            if code in self.kids:
                self.x_ang[code] = proc.n_out - 2 + 2 * len(self.x_ang)
                pre(self.kids[code][0])
                pre(self.kids[code][1])

        post(self.root)
        pre(self.root)

    def limits(self, code, sqrts):
        m_max = sqrts - self.m_min[self.root] + self.m_min[code]
        return self.m_min[code] ** 2, m_max * m_max, m_max

    def volume(self, sqrts):
        v = torch.ones_like(sqrts)
        for code in self.kids:
            v = v / (4 * (2 * math.pi) ** 5) if code == self.root else v * sqrts * sqrts / (4 * (2 * math.pi) ** 2)
        return v


def _msq_constants(t, m, w, mn, mx, s):
    if t == P.MAP_SCHANNEL:
        a0, a1 = torch.atan((mn - m * m) / (m * w)), torch.atan((mx - m * m) / (m * w))
        return a0, a1, (a1 - a0) * (m * w) / s
    if t in (P.MAP_RADIATION, P.MAP_COLLINEAR, P.MAP_INFRARED):
        a0 = w * w if t == P.MAP_RADIATION else m * m
        a1 = torch.log((mx - mn) / a0 + 1)
        return a0, a1, a1 / s
    if t in (P.MAP_TCHANNEL, P.MAP_UCHANNEL):
        a1 = 2 * torch.log((mx - mn) / (2 * m * m) + 1)
        return m * m, a1, a1 / s
    return None, None, (mx - mn) / s


def _msq_of_x(t, x, m, w, mn, mx, s):
    a0, a1, a2 = _msq_constants(t, m, w, mn, mx, s)
    if t == P.MAP_SCHANNEL:
        tz = torch.tan((1 - x) * a0 + x * a1)
        return m * (m + w * tz), a2 * (1 + tz * tz)
    if t in (P.MAP_RADIATION, P.MAP_COLLINEAR, P.MAP_INFRARED):
        q = a0 * torch.exp(x * a1)
        return q - a0 + mn, a2 * q
    if t in (P.MAP_TCHANNEL, P.MAP_UCHANNEL):
        q = a0 * torch.exp(torch.where(x < 0.5, x, 1 - x) * a1)
        return torch.where(x < 0.5, q - a0 + mn, -(q - a0) + mx), a2 * q
    return (1 - x) * mn + x * mx, a2 + torch.zeros_like(x)


def _x_of_msq(t, msq, m, w, mn, mx, s):
    a0, a1, a2 = _msq_constants(t, m, w, mn, mx, s)
    if t == P.MAP_SCHANNEL:
        z = (msq - m * m) / (m * w)
        return (torch.atan(z) - a0) / (a1 - a0), a2 * (1 + z * z)
    if t in (P.MAP_RADIATION, P.MAP_COLLINEAR, P.MAP_INFRARED):
        q = msq - mn + a0
        return torch.log(q / a0) / a1, a2 * q
    if t in (P.MAP_TCHANNEL, P.MAP_UCHANNEL):
        low = msq < (mx + mn) / 2
        q = torch.where(low, msq - mn, mx - msq) + a0
        lx = torch.log(q / a0) / a1
        return torch.where(low, lx, 1 - lx), a2 * q
    return (msq - mn) / (mx - mn), a2 + torch.zeros_like(msq)


_TWO_SIDED = (P.MAP_COLLINEAR, P.MAP_TCHANNEL, P.MAP_UCHANNEL)


def _ct_of_x(t, x, m, s):
    if t in _TWO_SIDED:
        b0 = m * m / s
        b1 = torch.log((b0 + 1) / b0)
        q = b0 * torch.exp(2 * torch.where(x < 0.5, x, 1 - x) * b1)
        ct = torch.where(x < 0.5, q - b0 - 1, -(q - b0) + 1)
        inside = (ct >= -1) & (ct <= 1)
        ct = torch.where(inside, ct, 1.0)
        st = torch.sqrt(torch.where(inside, 1 - ct * ct, 0.0))
        return ct, st, torch.where(inside, q * b1, 0.0)
    q = 2 * (1 - x)
    return 1 - q, torch.sqrt(q * (2 - q)), torch.ones_like(x)


def _x_of_ct(t, ct, m, s):
    if t in _TWO_SIDED:
        b0 = m * m / s
        b1 = torch.log((b0 + 1) / b0)
        q = torch.where(ct < 0, ct, -ct) + b0 + 1
        lx = torch.log(q / b0) / (2 * b1)
        return torch.where(ct < 0, lx, 1 - lx), q * b1
    return (ct + 1) / 2, torch.ones_like(ct)


def _lab(e1, e2):
    """sqrt(s), and the boost (beta gamma, gamma) along z, of beams e1, e2."""
    sqrts = 2 * torch.sqrt(e1 * e2)
    bg = (e1 - e2) / sqrts
    return sqrts, bg, torch.sqrt(1 + bg * bg)


def _events(tree, x, e1, e2, theta=None):
    """Momenta [n, n_out, 4], factor, volume and ok of one channel's events.  theta: mass and
    width per branch (tensors that gradients are wanted of)."""
    one = torch.ones(x.shape[0], dtype=torch.float64, device=x.device)
    sqrts, lab_bg, lab_ga = _lab(e1, e2)
    sqrts = sqrts * one
    s, zero = sqrts * sqrts, 0 * one
    msq, mass, factor, ok = {}, {}, one, torch.ones_like(one, dtype=torch.bool)
    par = {b: tuple(torch.as_tensor(v, dtype=torch.float64, device=x.device) for v in q[1:])
           for b, q in tree.map.items()}
    par.update(theta or {})
    for b, m in tree.leaf_m.items():
        msq[b], mass[b] = m * m * one, math.sqrt(m * m) * one
    msq[tree.root], mass[tree.root] = s, sqrts
    for b, k in tree.x_msq.items():
        mn, mx, m_max = tree.limits(b, sqrts)
        msq[b], f = _msq_of_x(tree.map[b][0], x[:, k], *par[b], mn + zero, mx, s)
        mass[b] = torch.sqrt(msq[b])
        factor = factor * f
        ok = ok & (mass[b] <= m_max)
    p = [None] * tree.n_out
    col = lambda *v: torch.stack(v, 1)  # noqa: E731
    lab = (col(lab_ga * one, zero, zero, lab_bg * one), col(zero, one, zero, zero),
           col(zero, zero, one, zero), col(lab_bg * one, zero, zero, lab_ga * one))
    todo = [(tree.root, lab, zero)]
    while todo:
        b, (c0, c1, c2, c3), pb = todo.pop()
        k = tree.kids[b]
        d = msq[b] - msq[k[0]] - msq[k[1]]
        lam = d * d - 4 * msq[k[0]] * msq[k[1]]
        ok = ok & (lam > 0) & (mass[b] > mass[k[0]] + mass[k[1]])
        root = torch.sqrt(lam)
        pd = root / (2 * mass[b])
        factor = factor * root / msq[b]
        bg = (pb / mass[b])[:, None]
        ga = torch.sqrt(1 + bg * bg)
        phi = 2 * math.pi * x[:, tree.x_ang[b]]
        ct, st, f = _ct_of_x(tree.map[b][0], x[:, tree.x_ang[b] + 1], par[b][0], s)
        factor = factor * f
        ct, st, cp, sp = (v[:, None] for v in (ct, st, torch.cos(phi), torch.sin(phi)))
        u, v, w = cp * c1 + sp * c2, cp * c2 - sp * c1, bg * c0 + ga * c3
        frame = (ga * c0 + bg * c3, ct * u - st * w, v, st * u + ct * w)
        for j, (code, sign) in enumerate(zip(k, (1, -1))):
            if code in tree.kids:
                todo.append((code, frame, sign * pd))
            else:
                e = torch.sqrt(msq[code] + pd * pd)
                p[code.bit_length() - 1] = frame[0] * e[:, None] + frame[3] * (sign * pd)[:, None]
    return torch.stack(p, 1), factor, tree.volume(sqrts), ok


def _pieces(proc, counts):
    """(channel, first, last) of runs of at most CHUNK events of one channel."""
    at = 0
    for c in range(proc.n_channels):
        for lo in range(at, at + int(counts[c]), CHUNK):
            yield c, lo, min(at + int(counts[c]), lo + CHUNK)
        at += int(counts[c])


def _forward(proc, counts, x, case, energies=None):
    out = [torch.zeros((x.shape[0], proc.n_out, 4), dtype=torch.float64, device=DEV),
           torch.zeros(x.shape[0], dtype=torch.float64, device=DEV),
           torch.zeros(x.shape[0], dtype=torch.float64, device=DEV),
           torch.zeros(x.shape[0], dtype=torch.uint8, device=DEV)]
    uniform = [torch.tensor(e, dtype=torch.float64, device=DEV) for e in _beams(case, proc)]
    for c, lo, hi in _pieces(proc, counts):
        e1, e2 = (e[lo:hi] for e in energies) if energies else uniform
        p, f, v, ok = _events(_Tree(proc, c), x[lo:hi], e1, e2)
        out[0][lo:hi] = torch.where(ok[:, None, None], p, 0.0)
        out[1][lo:hi] = torch.where(ok, f, 0.0)
        out[2][lo:hi] = v
        out[3][lo:hi] = ok
    return out


def _gradients(proc, x, pbar, jbar, case):
    tree = _Tree(proc, 0)
    uniform = [torch.tensor(e, dtype=torch.float64, device=DEV) for e in _beams(case, proc)]
    xbar = torch.zeros_like(x)
    thbar = torch.zeros((x.shape[0], max(1, proc.n_out - 2), 2), dtype=torch.float64, device=DEV)
    with torch.no_grad():
        ok = torch.cat([_events(tree, q, *uniform)[3] for q in x.split(CHUNK)])
    for at in torch.nonzero(ok)[:, 0].split(CHUNK // 4):
        xs = x[at].requires_grad_(True)
        theta = {b: tuple(torch.full((at.numel(),), v, dtype=torch.float64, device=DEV,
                                     requires_grad=True) for v in tree.map[b][1:])
                 for b in tree.x_msq if tree.map[b][0] == P.MAP_SCHANNEL}
        p, f, _, _ = _events(tree, xs, *uniform, theta)
        loss = (p * pbar[at]).sum() + (jbar[at] * torch.log(f)).sum()
        got = torch.autograd.grad(loss, [xs] + [v for q in theta.values() for v in q])
        xbar[at] = got[0]
        for i, b in enumerate(theta):
            thbar[at, tree.x_msq[b], 0] = got[1 + 2 * i]
            thbar[at, tree.x_msq[b], 1] = got[2 + 2 * i]
    return xbar, thbar


def _inverse(proc, counts, p, ok, x, factor, case):
    e1, e2 = (torch.tensor(e, dtype=torch.float64, device=DEV) for e in _beams(case, proc))
    sqrts, bg, ga = _lab(e1, e2)
    s = sqrts * sqrts
    cm = p.clone()
    if case["beams"] == "lab":
        cm[..., 0], cm[..., 3] = ga * p[..., 0] - bg * p[..., 3], ga * p[..., 3] - bg * p[..., 0]
    own = torch.repeat_interleave(torch.arange(proc.n_channels, device=DEV),
                                  torch.as_tensor(np.asarray(counts), device=DEV))
    all_f = torch.zeros((p.shape[0], proc.n_channels), dtype=torch.float64, device=DEV)
    all_x = torch.zeros((proc.n_channels, *x.shape), dtype=torch.float64, device=DEV)
    for c in range(proc.n_channels):
        f, xc = _inverse_channel(_Tree(proc, c), cm, sqrts, s, x.shape[1])
        mine, good = own == c, ok.bool()
        all_f[:, c] = torch.where(mine, factor, torch.where(good, f, 0.0))
        all_x[c] = torch.where(mine[:, None], x, torch.where(good[:, None], xc, 0.0))
    return all_f, all_x


def _inverse_channel(tree, cm, sqrts, s, n_x):
    q = {1 << j: cm[:, j] for j in range(tree.n_out)}

    def total(code):
        if code not in q:
            q[code] = total(tree.kids[code][0]) + total(tree.kids[code][1])
        return q[code]

    total(tree.root)
    minkowski = lambda v: v[:, 0] ** 2 - v[:, 1] ** 2 - v[:, 2] ** 2 - v[:, 3] ** 2  # noqa: E731
    msq = {b: minkowski(v) for b, v in q.items()}
    one = torch.ones(cm.shape[0], dtype=torch.float64, device=DEV)
    msq[tree.root] = s * one
    x = torch.zeros((cm.shape[0], n_x), dtype=torch.float64, device=DEV)
    factor = one
    # a frame: rows of the matrix that takes CM momenta to the branch's rest frame
    unit = torch.eye(4, dtype=torch.float64, device=DEV)
    todo = [(tree.root, [unit[i].expand(cm.shape[0], 4) for i in range(4)])]
    while todo:
        b, rows = todo.pop()
        t, m, w = tree.map[b]
        m = torch.tensor(m, dtype=torch.float64, device=DEV)
        k = tree.kids[b]
        for code in k:
            if code in tree.kids:
                tt, *mw = tree.map[code]
                mw = [torch.tensor(v, dtype=torch.float64, device=DEV) for v in mw]
                mn, mx, _ = tree.limits(code, sqrts)
                xm, f = _x_of_msq(tt, msq[code], *mw, mn, mx, s)
                x[:, tree.x_msq[code]] = xm
                factor = factor * f
        d = msq[b] - msq[k[0]] - msq[k[1]]
        root = torch.sqrt(d * d - 4 * msq[k[0]] * msq[k[1]])
        pd = root / (2 * torch.sqrt(msq[b]))
        factor = factor * root / msq[b]
        v = [(r * q[k[0]]).sum(1) for r in rows]
        phi = torch.atan2(v[2], v[1])
        phi = torch.where(phi < 0, phi + 2 * math.pi, phi)
        ct = v[3] / torch.sqrt(v[1] * v[1] + v[2] * v[2] + v[3] * v[3])
        st = torch.sqrt(1 - ct * ct)
        x[:, tree.x_ang[b]] = phi / (2 * math.pi)
        xc, f = _x_of_ct(t, ct, m, s)
        x[:, tree.x_ang[b] + 1] = xc
        factor = factor * f
        cp, sp, ct, st = (u[:, None] for u in (torch.cos(phi), torch.sin(phi), ct, st))
        for code, sign in zip(k, (1, -1)):
            if code in tree.kids:
                bg = (sign * pd / torch.sqrt(msq[code]))[:, None]
                ga = torch.sqrt(1 + bg * bg)
                u, w2 = cp * rows[1] + sp * rows[2], cp * rows[2] - sp * rows[1]
                z = st * u + ct * rows[3]
                todo.append((code, [ga * rows[0] - bg * z, ct * u - st * rows[3], w2,
                                    ga * z - bg * rows[0]]))
    return factor, x
