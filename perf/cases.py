"""Performance cases of the network update, through the package's entry points.

A case is one call that a program which uses this package makes: a simulation
advanced by some steps with its trace and its state read back, a batch of
networks advanced together, the allocation-free run on buffers of the caller,
a set of requests given to the server.  Topologies and states are drawn on the
GPU with torch, so that inputs are quick to make and come from the seed alone;
they have the shapes that the package's generators give: uniform density, a
grid with distance-dependent connections, a fixed number of random senders.

Conductances are kept below the explicit Euler step's limit of stability
(DELTA x degree x g well below 2): past it a network's voltages oscillate
without bound to their spread, and no two roundings of it agree.
"""
import ctypes as C
import math
import os

import numpy as np
import torch

import infoli_gb300 as ig

_CONF = os.path.join(os.path.dirname(os.path.abspath(ig.__file__)), "host", "default.conf")
_TRACES = {"axon": ig.TRACE_AXON, "soma": ig.TRACE_SOMA, "dend": ig.TRACE_DEND,
           "all": ig.TRACE_AXON | ig.TRACE_SOMA | ig.TRACE_DEND}
_G = 0.04          # the default conductance of an edge
_G_DEGREE = 25.0   # degree x g at most


def listed():
    return [
        # the smallest call: a few steps of a small network, every step traced
        dict(name="tiny50", kind="sim", topology="uniform", n=50, p=0.3, edge_g=False, kahan=False, steps=20,
             every=1, trace="axon", pulses="one"),
        # the reference's plain run: 1,000 cells at 10 % density, the axon printed every 100 steps
        dict(name="uniform1k", kind="sim", topology="uniform", n=1000, p=0.1, edge_g=False, kahan=True, steps=1000,
             every=100, trace="axon", pulses="none"),
        # the headline: 100 x 100 cells, Gaussian distance, about 440 senders a cell
        dict(name="grid10k", kind="sim", topology="grid", rows=100, cols=100, sigma=10.0, radius=18.0, edge_g=False,
             kahan=True, steps=1000, every=100, trace="axon", pulses="none"),
        # a grid of odd sides with a conductance per edge (as connectivity files give), all compartments traced
        dict(name="grid61x83_g", kind="sim", topology="grid", rows=61, cols=83, sigma=6.5, radius=12.0, edge_g=True,
             kahan=False, steps=500, every=50, trace="all", pulses="cells"),
        # 100,000 cells with 100 random senders each, a conductance per edge, a pulse of its own for each cell
        dict(name="sparse100k_g", kind="sim", topology="degree", n=100000, k=100, edge_g=True, kahan=True, steps=1000,
             every=500, trace="axon", pulses="cells"),
        # a sparse network of middle size with one conductance
        dict(name="sparse48k", kind="sim", topology="degree", n=48017, k=33, edge_g=False, kahan=False, steps=500,
             every=100, trace="soma", pulses="one"),
        # a dense network with one conductance, too large for a CTA's window and edges
        dict(name="dense10k", kind="sim", topology="uniform", n=10000, p=0.2, edge_g=False, kahan=True, steps=300,
             every=100, trace="axon", pulses="none"),
        # a dense matrix of conductances, as the connectivity files of the older simulator hold
        dict(name="dense6k_g", kind="sim", topology="uniform", n=6007, p=0.25, edge_g=True, kahan=False, steps=300,
             every=100, trace="axon", pulses="cells"),
        # the larger dense networks that are served
        dict(name="dense16k", kind="sim", topology="uniform", n=16000, p=0.3, edge_g=False, kahan=True, steps=200,
             every=100, trace="axon", pulses="one"),
        # many networks of uneven size and density in one launch
        dict(name="batch128", kind="batch", nets=128, lo=256, hi=8192, p_lo=0.05, p_hi=0.5, kahan=True, steps=200),
        # the allocation-free run on the caller's own device buffers
        dict(name="noalloc5k_g", kind="noalloc", n=5003, k=60, edge_g=True, steps=200, trace=True),
        # requests of uneven size and length, planned, run side by side and read back
        dict(name="serve6", kind="serve", requests=6, lo=500, hi=6000, p_lo=0.01, p_hi=0.3, steps_lo=400,
             steps_hi=1200, kahan=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Any of the listed kinds, over the ranges that they stand for; lengths are cut to a budget of work."""
    flag = lambda: rng.random() < 0.5  # noqa: E731
    kind = rng.choice(["small", "grid", "sparse", "dense", "dense_g", "batch", "noalloc", "serve"])
    trace, pulses = rng.choice(sorted(_TRACES)), rng.choice(["none", "one", "cells"])
    if kind == "batch":
        lo = _log(rng, 64, 1024)
        c = dict(kind="batch", nets=rng.randint(4, 96), lo=lo, hi=max(lo, _log(rng, 300, 8192)),
                 p_lo=rng.uniform(0.02, 0.2), p_hi=rng.uniform(0.2, 0.5), kahan=flag(), steps=_log(rng, 20, 300))
    elif kind == "noalloc":
        c = dict(kind="noalloc", n=_log(rng, 100, 20000), k=_log(rng, 8, 90), edge_g=flag(), steps=_log(rng, 10, 200),
                 trace=flag())
    elif kind == "serve":
        lo = _log(rng, 100, 1000)
        c = dict(kind="serve", requests=rng.randint(2, 6), lo=lo, hi=max(lo, _log(rng, 500, 6000)), p_lo=0.01,
                 p_hi=rng.uniform(0.05, 0.3), steps_lo=_log(rng, 100, 400), steps_hi=_log(rng, 400, 1200), kahan=flag())
    else:
        c = dict(kind="sim", kahan=flag(), edge_g=flag(), steps=_log(rng, 10, 1000), trace=trace, pulses=pulses)
        if kind == "small":
            c.update(topology="uniform", n=_log(rng, 10, 3000), p=rng.uniform(0.02, 0.5))
        elif kind == "grid":
            sigma = rng.uniform(2.0, 10.0)
            c.update(topology="grid", rows=_log(rng, 12, 100), cols=_log(rng, 12, 100), sigma=sigma, radius=1.8 * sigma)
        elif kind == "sparse":
            n = _log(rng, 3000, 100000)
            c.update(topology="degree", n=n, k=_log(rng, 8, 100))
        elif kind == "dense":
            c.update(topology="uniform", n=_log(rng, 5000, 16000), p=rng.uniform(0.07, 0.3), edge_g=False)
        else:
            c.update(topology="uniform", n=_log(rng, 3000, 7000), p=rng.uniform(0.1, 0.3), edge_g=True)
    budget = 0.9 * max(_cost(x) for x in listed())
    if "steps" in c and _cost(c) > budget:
        c["steps"] = max(1, int(c["steps"] * budget / _cost(c)))
    if c["kind"] == "sim":
        c["every"] = max(1, c["steps"] // rng.choice([1, 2, 5, 10]))
    return c


# ---------------------------------------------------------------------- work

def _means(case):
    """(cells, edges, steps) of a case, on average."""
    k = case["kind"]
    if k == "batch" or k == "serve":
        lo, hi = case["lo"], case["hi"]
        s = math.log(hi / lo) if hi > lo else 0.0
        m1 = (hi - lo) / s if s else lo
        m2 = (hi * hi - lo * lo) / (2 * s) if s else lo * lo
        cnt = case["nets"] if k == "batch" else case["requests"]
        steps = case["steps"] if k == "batch" else (case["steps_lo"] + case["steps_hi"]) / 2
        return cnt * m1, cnt * m2 * (case["p_lo"] + case["p_hi"]) / 2, steps
    if k == "noalloc" or case["topology"] == "degree":
        return case["n"], case["n"] * min(case["k"], case["n"] - 1), case["steps"]
    if case["topology"] == "uniform":
        return case["n"], case["n"] * (case["n"] - 1) * case["p"], case["steps"]
    rows, cols = case["rows"], case["cols"]
    e = 0.0
    R = int(case["radius"])
    for dr in range(-R, R + 1):
        for dc in range(-R, R + 1):
            d2 = dr * dr + dc * dc
            if 0 < d2 <= case["radius"] ** 2:
                e += max(0, rows - abs(dr)) * max(0, cols - abs(dc)) * math.exp(-d2 / (2 * case["sigma"] ** 2))
    return rows * cols, e, case["steps"]


def work(case):
    """Each edge once per step: a difference, its square, an exponential, the weight and the sum (8 operations,
    the exponential counted as one), 300 per cell for its gates, currents and voltages.  Bytes: the topology (a
    bit per ordered pair where it is passed as bits, else a sender id and a conductance, if any, per edge), the 19
    state arrays in and out, the trace."""
    n, e, steps = _means(case)
    edge = 8.0 if case.get("edge_g") else 4.0
    topo = e / ((case["p_lo"] + case["p_hi"]) / 2) / 8 if case["kind"] == "batch" else e * edge
    rows = 0
    if case["kind"] == "sim":
        rows = len(range(0, case["steps"], case["every"])) * (3 if case["trace"] == "all" else 1) if "every" in case else 0
    elif case["kind"] == "noalloc" and case["trace"]:
        rows = steps
    return {"bytes": topo + n * (2 * 19 + rows) * 4.0, "flops": steps * (8.0 * e + 300.0 * n)}


def _cost(case):
    return work(case)["flops"]


# -------------------------------------------------------------------- inputs

def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _conf():
    return np.array([float(s.split("=")[1]) for s in open(_CONF) if "=" in s], dtype=np.float32)


def _rand(gen, shape, lo, hi):
    return torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo


def _state(gen, conf, n):
    """[19, n]: the defaults, V_dend spread by a millivolt about rest, g_CaL uniform in 0.6 to 0.8."""
    st = torch.from_numpy(conf[23:42].copy()).cuda()[:, None].repeat(1, n)
    st[0] += _rand(gen, n, -1.0, 1.0)
    st[6] = _rand(gen, n, 0.6, 0.8)
    return st


def _rows_of(mask_rows, n):
    """CSR on the GPU from an iterator over blocks of rows of a boolean matrix."""
    counts, cols = [], []
    for m in mask_rows:
        counts.append(m.sum(1))
        cols.append(m.nonzero()[:, 1].to(torch.int32))
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cat(counts).cumsum(0)
    return rp, torch.cat(cols)


def _uniform_blocks(gen, n, p):
    step = max(1, (1 << 27) // n)
    for r0 in range(0, n, step):
        r1 = min(n, r0 + step)
        m = torch.rand((r1 - r0, n), generator=gen, device="cuda") < p
        m[torch.arange(r1 - r0, device="cuda"), torch.arange(r0, r1, device="cuda")] = False
        yield m


def _degree(gen, n, k):
    """n rows of k distinct senders, ascending, none of them the row itself."""
    k = min(k, n - 1)
    ids = torch.randint(0, n - k, (n, k), generator=gen, device="cuda").sort(1)[0] + torch.arange(k, device="cuda")
    ids += ids >= torch.arange(n, device="cuda")[:, None]
    return torch.arange(0, n * k + 1, k, device="cuda"), ids.reshape(-1).to(torch.int32)


def _grid(gen, rows, cols, sigma, radius):
    R = int(radius)
    d = [(a, b) for a in range(-R, R + 1) for b in range(-R, R + 1) if 0 < a * a + b * b <= radius * radius]
    off = torch.tensor(d, device="cuda")
    prob = torch.exp(-(off.double() ** 2).sum(1) / (2 * sigma * sigma)).float()
    n = rows * cols
    i = torch.arange(n, device="cuda")
    r, c = (i // cols)[:, None] + off[:, 0], (i % cols)[:, None] + off[:, 1]
    hit = (torch.rand((n, len(d)), generator=gen, device="cuda") < prob) & (r >= 0) & (r < rows) & (c >= 0) & (c < cols)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = hit.sum(1).cumsum(0)
    return rp, (r * cols + c)[hit].to(torch.int32)


def _network(case, gen):
    """(n, row_ptr, col, g or None, one conductance) on the GPU."""
    if case["kind"] == "noalloc" or case["topology"] == "degree":
        n = case["n"]
        rp, col = _degree(gen, n, case["k"])
    elif case["topology"] == "uniform":
        n = case["n"]
        rp, col = _rows_of(_uniform_blocks(gen, n, case["p"]), n)
    else:
        n = case["rows"] * case["cols"]
        rp, col = _grid(gen, case["rows"], case["cols"], case["sigma"], case["radius"])
    g1 = min(_G, _G_DEGREE / max(1.0, col.numel() / n))
    g = _rand(gen, col.numel(), 0.5 * g1, 1.5 * g1) if case["edge_g"] else None
    return n, rp, col, g, float(np.float32(g1))


def _spread(count):
    """`count` points that fill the unit cube evenly: sizes, densities and conductances (or lengths) of the networks
    of one case, the same for every seed, the sizes ragged and out of order."""
    return [((i * 0.6180339887 + 0.5) % 1.0, (i * 0.7548776662 + 0.25) % 1.0, (i * 0.5698402910 + 0.75) % 1.0)
            for i in range(count)]


def _batch_networks(case, gen):
    """Per network (cells, row_ptr, col, bits as the package takes them, conductance)."""
    nets = []
    for a, b, c in _spread(case["nets"]):
        n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** a))
        p = case["p_lo"] + (case["p_hi"] - case["p_lo"]) * b
        w = (n + 31) // 32
        bits = torch.zeros((n, w), dtype=torch.int64, device="cuda")
        m = torch.zeros((n, w * 32), dtype=torch.bool, device="cuda")
        m[:, :n] = torch.cat(list(_uniform_blocks(gen, n, p)))
        for k in range(32):
            bits |= m[:, k::32].long() << k
        rp, col = _rows_of([m], n)
        nets.append((n, rp, col, bits, float(np.float32(min(0.02 + 0.04 * c, _G_DEGREE / (n * p + 1))))))
    return nets


def _pulses(case, gen, n):
    """None, one pulse (start, end, amplitude) for all cells, or (amplitude, onset, duration) per cell."""
    steps = case["steps"]
    if case["pulses"] == "none":
        return None
    if case["pulses"] == "one":
        return (steps // 4, steps // 2 + 1, 1.0)  # below the threshold: a spike would blow up roundings
    return (_rand(gen, n, 0.0, 8.0), torch.randint(0, steps, (n,), generator=gen, device="cuda").int(), 100)


def _requests(case, gen):
    out = []
    for a, b, c in _spread(case["requests"]):
        n = int(round(case["lo"] * (case["hi"] / case["lo"]) ** a))
        p = case["p_lo"] + (case["p_hi"] - case["p_lo"]) * b
        steps = int(round(case["steps_lo"] + (case["steps_hi"] - case["steps_lo"]) * c))
        rp, col = _rows_of(_uniform_blocks(gen, n, p), n)
        g = float(np.float32(min(_G, _G_DEGREE / (n * p + 1))))
        out.append((n, rp, col, g, steps))
    return out


def _host(t):
    return None if t is None else t.cpu().numpy()


# ----------------------------------------------------------------- the calls

def prepare(case, seed):
    gen, conf = _rng(seed), _conf()
    kind = case["kind"]
    if kind == "batch":
        nets = _batch_networks(case, gen)
        st = _state(gen, conf, sum(x[0] for x in nets))
        sizes = [(n, _host(bits).astype(np.uint32), g) for n, _, _, bits, g in nets]
        return {"kind": kind, "steps": case["steps"],
                "batch": ig.Batch(conf, sizes, init_state=_host(st), kahan=case["kahan"])}
    if kind == "serve":
        reqs = [(n, _host(rp), _host(col), g, steps, _host(_state(gen, conf, n)))
                for n, rp, col, g, steps in _requests(case, gen)]
        return {"kind": kind, "reqs": reqs, "server": ig.Server(conf, kahan=case["kahan"])}
    n, rp, col, g, g1 = _network(case, gen)
    if kind == "noalloc":
        st = _state(gen, conf, n).reshape(-1).contiguous()
        tr = torch.zeros(case["steps"] * n, device="cuda") if case["trace"] else None
        return {"kind": kind, "n": n, "rp": rp, "col": col, "g": g, "g1": g1, "state": st, "trace": tr,
                "steps": case["steps"], "at": 0, "params": conf[:23].copy()}
    st = _state(gen, conf, n)
    pulse = _pulses(case, gen, n)
    sim = ig.Simulation(n, conf, _host(rp), _host(col), g=_host(g), g_uniform=g1, init_state=_host(st),
                        kahan=case["kahan"])
    if case["pulses"] == "one":
        sim.set_stimulus_pulse(*pulse)
    elif case["pulses"] == "cells":
        sim.set_stimulus_cells(_host(pulse[0]), _host(pulse[1]), pulse[2])
    return {"kind": kind, "sim": sim, "steps": case["steps"], "every": case["every"], "what": _TRACES[case["trace"]]}


def run(state):
    kind = state["kind"]
    if kind == "sim":
        out = state["sim"].run(state["steps"], state["every"], state["what"])
        out["state"] = state["sim"].get_state()
        return out
    if kind == "batch":
        state["batch"].run(state["steps"])
        return state["batch"].get_state()
    if kind == "serve":
        sv = state["server"]
        ids = [sv.submit(n, rp, col, steps, g_uniform=g, init_state=st) for n, rp, col, g, steps, st in state["reqs"]]
        return [sv.wait(i)[0] for i in ids]
    ptr = lambda t: None if t is None else C.c_void_p(t.data_ptr())  # noqa: E731
    lib = ig.capi.load()
    rc = lib.infoli_run_noalloc(state["params"].ctypes.data_as(C.c_void_p), state["n"], ptr(state["rp"]),
                                ptr(state["col"]), ptr(state["g"]), state["g1"], 50, 120, 6.0, ptr(state["state"]),
                                state["at"], state["steps"], ptr(state["trace"]),
                                C.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError(lib.infoli_last_error().decode())
    state["at"] += state["steps"]
    return [state["state"]] + ([state["trace"]] if state["trace"] is not None else [])


# -------------------------------------------------------------- 64-bit values

def _cell(P, s, ic, iapp):
    """One explicit Euler step of every cell, in 64 bits: gates first, all derivatives from the old voltages."""
    (dt, _, cm, gna, gkdr, gks, gls, gkca, gcah, gld, gh, gnaa, _, gka, gla, p1, p2, gint, vna, vk, vca, vh, vl) = P
    e = torch.exp
    Vd, Vs, Va, Ca, ICaH = s[0], s[7], s[15], s[4], s[5]
    q = s[3] + dt * (1 / (1 + e((Vd + 80) / 4)) - s[3]) * (e(-0.086 * Vd - 14.6) + e(0.070 * Vd - 1.87))
    ar = 1.7 / (1 + e(-(Vd - 5) / 13.9))
    br = 0.02 * (Vd + 8.5) / (e((Vd + 8.5) / 5) - 1)
    r = s[1] + dt * (ar / (ar + br) - s[1]) * (ar + br) / 5
    a_s = torch.clamp(0.00002 * Ca, max=0.01)
    ss = s[2] + dt * (a_s / (a_s + 0.015) - s[2]) * (a_s + 0.015)
    ca = Ca + dt * (-3 * ICaH - 0.075 * Ca)
    icah = gcah * r * r * (Vd - vca)
    dVd = -(icah + gint / (1 - p1) * (Vd - Vs) + gld * (Vd - vl) + gkca * ss * (Vd - vk) + ic + gh * q * (Vd - vh)) + iapp
    k = s[13] + dt * (1 / (1 + e(-(Vs + 61) / 4.2)) - s[13])
    tl = 20 * e((Vs + 160) / 30) / (1 + e((Vs + 84) / 7.3)) + 35
    l = s[14] + dt * (1 / (1 + e((Vs + 85.5) / 8.5)) - s[14]) / tl
    m = 1 / (1 + e((-30 - Vs) / 5.5))
    h = s[9] + dt * (1 / (1 + e((70 + Vs) / 5.8)) - s[9]) / (3 * e((-40 - Vs) / 33))
    tn = 5 + 47 * e((50 + Vs) / 900)
    n = s[10] + dt * (1 / (1 + e((-3 - Vs) / 10)) - s[10]) / tn
    p = s[11] + dt * (1 / (1 + e((51 + Vs) / 12)) - s[11]) / tn
    ax, bx = 0.13 * (Vs + 25) / (1 - e(-(Vs + 25) / 10)), 1.69 * e(-0.0125 * (Vs + 35))
    x = s[12] + 0.05 * (ax / (ax + bx) - s[12]) * (ax + bx)
    dVs = -(s[6] * k ** 3 * l * (Vs - vca) + gint / p1 * (Vs - Vd) + gint / (1 - p2) * (Vs - Va)
            + gna * m ** 3 * h * (Vs - vna) + gls * (Vs - vl) + gkdr * n ** 4 * (Vs - vk) + gks * x ** 4 * (Vs - vk))
    ma = 1 / (1 + e((-30 - Va) / 5.5))
    ha = s[17] + dt * (1 / (1 + e((60 + Va) / 5.8)) - s[17]) / (1.5 * e((-40 - Va) / 33))
    ay, by = 0.13 * (Va + 25) / (1 - e(-(Va + 25) / 10)), 1.69 * e(-0.0125 * (Va + 35))
    xa = s[18] + 0.05 * (ay / (ay + by) - s[18]) * (ay + by)
    dVa = -(gka * xa ** 4 * (Va - vk) + gint / p2 * (Va - Vs) + gla * (Va - vl) + gnaa * ma ** 3 * ha * (Va - vna))
    return torch.stack([Vd + dt * dVd / cm, r, ss, q, ca, icah, s[6], Vs + dt * dVs / cm, m, h, n, p, x, k, l,
                        Va + dt * dVa / cm, ma, ha, xa])


def _advance(conf, st, rp, col, g, steps, every=0, rows=(), iapp=None):
    """(state, {row name: [rows, n]}) after `steps` steps in 64 bits; g: per edge, or one number."""
    P = [float(v) for v in conf[:23].astype(np.float64)]
    s = st.double()
    n = s.shape[1]
    dst = torch.repeat_interleave(torch.arange(n, device="cuda"), rp[1:] - rp[:-1])
    col = col.long()
    g = g.double() if torch.is_tensor(g) else float(g)
    none = torch.zeros(n, dtype=torch.float64, device="cuda")
    got = {k: [] for k in rows}
    at = {"axon": 15, "soma": 7, "dend": 0}
    for t in range(steps):
        V = s[0][dst] - s[0][col]
        f = V * V
        f.mul_(-0.01).exp_().mul_(0.8).add_(0.2).mul_(V).mul_(g)
        ic = torch.segment_reduce(f, "sum", offsets=rp, initial=0.0)
        s = _cell(P, s, ic, none if iapp is None else iapp(t))
        if every and t % every == 0:
            for k in rows:
                got[k].append(s[at[k]].clone())
    return s, {k: torch.stack(v) for k, v in got.items()}


def exact(case, seed):
    gen, conf = _rng(seed), _conf()
    kind = case["kind"]
    if kind == "batch":
        nets = _batch_networks(case, gen)
        if sum(x[2].numel() for x in nets) * case["steps"] > 1.2e11:
            return None
        st = _state(gen, conf, sum(x[0] for x in nets))
        off = np.concatenate([[0], np.cumsum([x[0] for x in nets])]).tolist()
        base = np.concatenate([[0], np.cumsum([x[2].numel() for x in nets])]).tolist()
        rp = torch.cat([x[1][:-1] + b for x, b in zip(nets, base)] + [torch.tensor([base[-1]], device="cuda")])
        col = torch.cat([x[2].long() + o for x, o in zip(nets, off)])
        g = torch.cat([torch.full((x[2].numel(),), x[4], dtype=torch.float64, device="cuda") for x in nets])
        return _advance(conf, st, rp, col, g, case["steps"])[0].cpu().numpy()
    if kind == "serve":
        return [_advance(conf, _state(gen, conf, n), rp, col, g, steps)[0].cpu().numpy()
                for n, rp, col, g, steps in _requests(case, gen)]
    n, rp, col, g, g1 = _network(case, gen)
    if col.numel() * case["steps"] > 1.2e11:
        return None
    st = _state(gen, conf, n)
    if kind == "noalloc":
        one = torch.full((n,), 6.0, dtype=torch.float64, device="cuda")
        s, tr = _advance(conf, st, rp, col, g if g is not None else g1, case["steps"], 1, ("axon",),
                         lambda t: one if 50 <= t < 120 else one * 0)
        return [s.reshape(-1)] + ([tr["axon"].reshape(-1)] if case["trace"] else [])
    pulse = _pulses(case, gen, n)
    iapp = None
    if case["pulses"] == "one":
        iapp = lambda t: torch.full((n,), pulse[2] if pulse[0] <= t < pulse[1] else 0.0, dtype=torch.float64, device="cuda")  # noqa: E731
    elif case["pulses"] == "cells":
        amp, on = pulse[0].double(), pulse[1].long()
        iapp = lambda t: amp * ((on <= t) & (t < on + pulse[2]))  # noqa: E731
    rows = [k for k in ("axon", "soma", "dend") if case["trace"] in (k, "all")]
    s, tr = _advance(conf, st, rp, col, g if g is not None else g1, case["steps"], case["every"], rows, iapp)
    tr["state"] = s
    return tr
