"""The work a program has this framework do, as cases to be timed and checked.

Every case goes through the public entry points: an `Fa2` handle advanced by a
few ticks with every tick's positions kept on the GPU, the registry's one-shot
call, a `Batch`, a recorded run and its backward pass, a live `ForceSession` on
the tree or on the particle mesh, and the layout's Kruskal stress. Sizes are
those of the workload recipes in `graph_render_b200.synth` and
`graph_render_b200.batch` and of the reference's benchmark model, and ragged
ones in between. `exact` restates a case in FP64 with plain torch: a quadtree or
octree walked level by level, the FA2 tick (differentiable, so the backward
pass's value is its gradient), the d3-force tick and the particle mesh.
"""

import math

import numpy as np
import torch

import graph_render_b200 as gr
from graph_render_b200 import batch, stress, synth

DEV = "cuda"


# ------------------------------------------------------------------ the cases --

def listed():
    return [
        # a live drawing of a small network: the smallest call, a few frames at a time
        dict(name="fa2_sbm_1500", kind="fa2", model="sbm", n=1500, dim=2, theta=1.2, opts="", ticks=8),
        # an ordinary graph at the reference's own default angle, a size off every power of two
        dict(name="fa2_gate_12345", kind="fa2", model="gate", n=12345, dim=2, theta=0.8, opts="", ticks=2),
        # a scale-free network with weights, log attraction and hubs dissuaded
        dict(name="fa2_ba_100k", kind="fa2", model="ba", n=100_000, dim=2, theta=1.0, opts="ldw", ticks=2),
        # the largest graphs, in the plane and in space
        dict(name="fa2_powerlaw_1m_2d", kind="fa2", model="powerlaw", n=1_000_000, dim=2, theta=1.2, opts="", ticks=2),
        dict(name="fa2_powerlaw_1m_3d", kind="fa2", model="powerlaw", n=1_000_000, dim=3, theta=1.2, opts="s", ticks=2),
        # a new graph laid out in one registry call from its seeded start: a first look after the
        # iterations that the reference compares its runs over
        dict(name="call_ba_4999", kind="call", model="ba", n=4999, theta=0.8, ticks=2),
        # many small networks at once
        dict(name="batch_512", kind="batch", graphs=512, nmin=50, nmax=20_000, ticks=2),
        # a gradient step on start positions and edge weights
        dict(name="backward_sbm_50k", kind="backward", n=50_000, theta=1.2),
        # a live d3-force drawing: tick, read the frame; small and largest
        dict(name="force_3001", kind="force", model="ba", n=3001, mesh=False, ticks=2),
        dict(name="force_1m", kind="force", model="gate", n=1_000_000, mesh=False, ticks=2),
        # the same drawing with its many-body pass on the particle mesh
        dict(name="mesh_300k", kind="force", model="gate", n=300_007, mesh=True, ticks=2),
        # a finished layout's quality
        dict(name="stress_200k", kind="stress", model="powerlaw", n=200_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fa2", "fa2", "fa2", "fa2", "call", "batch", "backward", "force", "force", "mesh", "stress"])
    if kind == "fa2":
        dim = rng.choice([2, 2, 3])
        opts = "".join(c for c in "ldws" if rng.random() < 0.3)
        return dict(kind="fa2", model=rng.choice(["gate", "ba", "powerlaw", "sbm"]), n=_log_int(rng, 300, 700_000), dim=dim,
                    theta=round(rng.uniform(0.7, 1.3), 2), opts=opts, ticks=rng.choice([1, 2]))
    if kind == "call":
        return dict(kind="call", model=rng.choice(["gate", "ba", "powerlaw"]), n=_log_int(rng, 500, 300_000),
                    theta=round(rng.uniform(0.7, 1.3), 2), ticks=rng.choice([1, 2]))
    if kind == "batch":
        return dict(kind="batch", graphs=_log_int(rng, 32, 512), nmin=rng.choice([50, 200]), nmax=_log_int(rng, 1000, 20_000),
                    ticks=rng.choice([1, 2]))
    if kind == "backward":
        return dict(kind="backward", n=_log_int(rng, 1000, 50_000), theta=round(rng.uniform(0.8, 1.2), 2))
    if kind == "stress":
        return dict(kind="stress", model=rng.choice(["gate", "ba", "powerlaw"]), n=_log_int(rng, 1000, 200_000))
    n = _log_int(rng, 500, 600_000)
    return dict(kind="force", model=rng.choice(["gate", "ba"]) if n < 10_000 else "gate", n=n, mesh=kind == "mesh", ticks=rng.choice([1, 2]))


# ------------------------------------------------------------------ the inputs --

def _graph(model, n, seed):
    """(source, target, weight) of one graph of a workload recipe, drawn from the seed."""
    if model == "sbm":  # four equal blocks, mean degree about 8
        sizes = [n // 4 + (1 if b < n % 4 else 0) for b in range(4)]
        p_in = min(1.0, 30.0 / n)
        src, dst = synth.sbm(sizes, p_in, min(1.0, p_in / 20.0), seed)
    elif model == "ba":
        src, dst = synth.ba(n, 3, seed)
    elif model == "gate":  # the reference's benchmark model is one graph per size: its nodes are renumbered
        src, dst, _ = synth.gate(n)
        perm = np.random.default_rng(seed).permutation(n).astype(np.uint32)
        src, dst = perm[src], perm[dst]
    else:
        src, dst = synth.config_powerlaw(n, seed)
    return src, dst, synth.lognormal(len(src), 0.0, 0.5, seed + 7)


def _start(model, n, dim, seed):
    if model == "sbm":
        return synth.uniform(n, dim, -1000.0, 1000.0, seed + 1000)
    side = 1e4 if model == "powerlaw" else math.sqrt(n) * 10.0
    return synth.uniform(n, dim, 0.0, side, seed + 1000)


def _fa2_params(case, seed):
    o = case.get("opts", "")
    return dict(theta=case["theta"], dim=case.get("dim", 2), seed=seed % (1 << 32), max_iter=max(case["ticks"], 1),
                lin_log=int("l" in o), dissuade_hubs=int("d" in o), edge_weight_influence=1.0 if "w" in o else 0.0,
                strong_gravity=int("s" in o))


def _fa2_inputs(case, seed):
    src, dst, w = _graph(case["model"], case["n"], seed)
    return src, dst, w if "w" in case["opts"] else None, _start(case["model"], case["n"], case["dim"], seed)


def _batch_inputs(case, seed):
    """The mixed batch (`batch.mixed_graph`'s kinds, options and start), its node counts evenly spread over
    their logarithm instead of drawn, so that another seed's batch has as many nodes."""
    out, graphs = [], case["graphs"]
    for i in range(graphs):
        r = np.random.default_rng([seed, i])
        n = int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** ((i + 0.5) / graphs)))
        kind, s = ("sbm", "ba", "grid")[int(r.integers(0, 3))], int(r.integers(0, 2 ** 62))
        if kind == "sbm":
            blocks, kbar = int(r.integers(2, 9)), float(r.uniform(4.0, 10.0))
            sizes = [n // blocks + (1 if b < n % blocks else 0) for b in range(blocks)]
            p_in = kbar / ((n / blocks - 1) + (n - n / blocks) / 20.0)
            src, dst = synth.sbm(sizes, min(1.0, p_in), min(1.0, p_in / 20.0), s)
        elif kind == "ba":
            src, dst = synth.ba(n, int(r.integers(2, 5)), s)
        else:
            src, dst = synth.grid(n, 0.05, s)
        prm = dict(scaling_ratio=float(r.uniform(1.0, 10.0)), gravity=float(r.uniform(0.1, 5.0)), theta=1.2, dim=2,
                   seed=int(r.integers(0, 2 ** 31)), max_iter=case["ticks"])
        out.append(batch.GraphSpec(n, src, dst, prm, None, synth.uniform(n, 2, 0.0, math.sqrt(n) * 10.0, s + 1), kind))
    return out


def _backward_inputs(case, seed):
    n = case["n"]
    scale = 50_000 / n
    sizes = [n // 16 + (1 if b < n % 16 else 0) for b in range(16)]
    # the differentiated workload's blocks at a mean degree of 16
    src, dst = synth.sbm(sizes, min(1.0, 5e-3 * scale), min(1.0, 5e-5 * scale), seed)
    keep = np.sort(np.random.default_rng(seed + 4).permutation(len(src))[:8 * n])  # as many edges whatever the seed
    src, dst = src[keep], dst[keep]
    w = synth.lognormal(len(src), 0.0, 0.25, seed + 7)
    pos = synth.uniform(n, 2, 0.0, math.sqrt(n) * 10.0, seed + 1000)
    grad = np.random.default_rng(seed + 2).standard_normal((n, 2)).astype(np.float32)
    return src, dst, w, pos, grad


def _force_inputs(case, seed):
    src, dst, _ = _graph(case["model"], case["n"], seed)
    return src, dst, np.random.default_rng(seed + 3).uniform(0.4, 0.8, len(src))


def _stress_inputs(case, seed):
    src, dst, _ = _graph(case["model"], case["n"], seed)
    p = synth.uniform(case["n"], 2, 0.0, 1e3, seed + 1000)
    return src, dst, np.ascontiguousarray(p[:, 0]), np.ascontiguousarray(p[:, 1])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fa2":
        src, dst, w, pos = _fa2_inputs(case, seed)
        eng = gr.Fa2(case["n"], src, dst, w, params=_fa2_params(case, seed), pos0=pos)
        out = torch.empty((case["ticks"], case["n"], case["dim"]), dtype=torch.float32, device=DEV)
        return dict(kind=kind, eng=eng, ticks=case["ticks"], out=out)
    if kind == "call":
        src, dst, w = _graph(case["model"], case["n"], seed)
        return dict(kind=kind, topology=gr.Topology(case["n"], src, dst, w), row=gr.find(gr.FA2_ID),
                    params=gr.fa2.params_bytes(_fa2_params(case, seed)))
    if kind == "batch":
        return dict(kind=kind, batch=batch.Batch(_batch_inputs(case, seed)), ticks=case["ticks"])
    if kind == "backward":
        src, dst, w, pos, grad = _backward_inputs(case, seed)
        eng = gr.Fa2(case["n"], src, dst, w, params=dict(theta=case["theta"], dim=2, seed=1, max_iter=1, edge_weight_influence=1.0),
                     pos0=pos)
        return dict(kind=kind, eng=eng, pos=pos, grad=grad)
    if kind == "force":
        src, dst, st = _force_inputs(case, seed)
        session = gr.ForceSession(case["n"], src, dst, st)
        if case["mesh"]:
            session.use_mesh()
        return dict(kind=kind, session=session, ticks=case["ticks"])
    src, dst, x, y = _stress_inputs(case, seed)
    return dict(kind=kind, src=src, dst=dst, x=x, y=y)


# -------------------------------------------------------------------- one pass --

def run(state):
    kind = state["kind"]
    if kind == "fa2":  # the next ticks, every tick's positions into a device buffer
        state["eng"].tick_record(state["ticks"], state["out"].data_ptr())
        return state["out"]
    if kind == "call":
        g = state["row"].run_params(state["topology"], state["params"])
        return np.asarray(g.x), np.asarray(g.y)
    if kind == "batch":
        state["batch"].run(state["ticks"])
        return np.concatenate(state["batch"].positions())
    if kind == "backward":
        # an optimiser's step: its present start positions in, a fresh controller, one tick
        # recorded, the gradients back (kept in FP32, as its positions and weights are)
        eng = state["eng"]
        eng.set_positions(state["pos"])
        eng.set_controller(1.0, 1.0, 1.0, 1.0, 0)
        eng.adjoint_forward(1, every=1)
        dp0, dw = eng.adjoint_backward(state["grad"])
        return dp0.astype(np.float32), dw.astype(np.float32)
    if kind == "force":
        s = state["session"]
        s.tick(state["ticks"])
        return s.positions(), s.velocities()
    return stress.kruskal_stress(state["x"], state["y"], state["src"], state["dst"])


def work(case):
    """Bytes: the graph, the positions in and out once a tick; operations: about 70 interactions a
    node (9 in the nearest ring and 3 a level above it at theta 1.2, more at smaller angles), 10
    operations each, and 6 a directed edge."""
    kind, t = case["kind"], case.get("ticks", 1)
    n = case.get("n", 0)
    if kind == "batch":
        lo, hi = case["nmin"], case["nmax"]
        n = case["graphs"] * (hi - lo) / math.log(hi / lo)
    deg = {"sbm": 8, "ba": 6, "gate": 3.1, "powerlaw": 8}.get(case.get("model", ""), 8 if kind != "backward" else 16)
    if kind == "stress":
        return {"bytes": n * (4 * deg + 8 + 8) + 16 * n, "flops": 16 * n * 10}
    near = 70 * (1.2 / case.get("theta", 0.9)) ** 2
    per = near * 10 + deg * 6 + 40
    byts = deg * 4 + 4 + 16 * 2 + 8
    if kind == "backward":
        per, byts = 3 * per, 3 * byts
    if kind == "force" and case["mesh"]:
        side = min(1024, max(128, 1 << math.ceil(math.log2(math.sqrt(n)))))
        per = 200 + 30 * side * side * math.log2(side) / n
        byts += 48 * side * side / n
    return {"bytes": byts * n * t, "flops": per * n * t}


# ---------------------------------------------------- the same in FP64, by torch --

def _f32(v):
    return float(np.float32(v))


def _seg(index, values, size):
    return torch.zeros((size,) + values.shape[1:], dtype=values.dtype, device=values.device).index_add(0, index, values)


def _keys(p, gid, graphs, levels):
    """Morton keys in each graph's root square (corner floor(min), side a power of two >= 1 that holds the maximum)."""
    dim = p.shape[1]
    lo = torch.full((graphs, dim), math.inf, dtype=p.dtype, device=p.device).index_reduce(0, gid, p, "amin")
    hi = torch.full((graphs, dim), -math.inf, dtype=p.dtype, device=p.device).index_reduce(0, gid, p, "amax")
    corner = lo.floor()
    side = torch.ones(graphs, dtype=p.dtype, device=p.device)
    for _ in range(200):
        grow = (hi >= corner + side[:, None]).any(1)
        if not grow.any():
            break
        side = torch.where(grow, side * 2, side)
    q = ((p - corner[gid]) / side[gid][:, None] * 2.0 ** levels).floor().clamp(0, 2 ** levels - 1).long()
    key = torch.zeros(len(p), dtype=torch.long, device=p.device)
    for b in range(levels):
        for a in range(dim):
            key |= ((q[:, a] >> b) & 1) << (b * dim + a)
    return key, side


def _walk(p, mass, gid, graphs, far_rule, body):
    """Sum over every node's tree walk of body(nodes, displacement to the node from the body's centre, body mass).

    far_rule(width, d2, holds) says where a cell acts as one body; a cell of one point always does (its own
    point excepted). Levels are visited in turn with the (node, cell) pairs that are still open."""
    n, dim = p.shape
    levels = 31 if dim == 2 else 20
    with torch.no_grad():
        key, side = _keys(p, gid, graphs, levels)
        order = torch.argsort(key, stable=True)
        order = order[torch.argsort(gid[order], stable=True)]
        key, g = key[order], gid[order]
    q, m = p[order], mass[order]
    me = torch.arange(n, device=p.device)
    total = torch.zeros_like(p)
    nodes, cells = me, g.clone()
    for level in range(levels + 1):
        with torch.no_grad():
            prefix = key >> (dim * (levels - level))
            new = torch.ones(n, dtype=torch.bool, device=p.device)
            new[1:] = (prefix[1:] != prefix[:-1]) | (g[1:] != g[:-1])
            of = torch.cumsum(new, 0) - 1
            first = torch.nonzero(new).squeeze(1)
            size = torch.diff(first, append=torch.tensor([n], device=p.device))
            if level == 0:
                cells = of[nodes]
        cm = _seg(of, m, len(first))
        cc = _seg(of, q * m[:, None], len(first)) / cm[:, None]
        with torch.no_grad():
            d2 = ((q[nodes] - cc[cells]) ** 2).sum(1)
            holds = of[nodes] == cells
            one = size[cells] == 1
            far = far_rule((side[g[nodes]] * 2.0 ** -level) ** 2, d2, holds) & ~one
            take = far | (one & ~holds)
            i, c = nodes[take], cells[take]
        total = total.index_add(0, i, body(order[i], q[i] - cc[c], cm[c]))
        with torch.no_grad():
            still = ~(far | one)
            nodes, cells = nodes[still], cells[still]
            if level == levels or len(nodes) == 0:
                break
            nxt = key >> (dim * (levels - level - 1))
            new2 = torch.ones(n, dtype=torch.bool, device=p.device)
            new2[1:] = (nxt[1:] != nxt[:-1]) | (g[1:] != g[:-1])
            of2 = torch.cumsum(new2, 0) - 1
            child = of2[first]
            count = torch.diff(child, append=(of2[-1:] + 1))[cells]
            at = torch.repeat_interleave(torch.arange(len(cells), device=p.device), count)
            within = torch.arange(len(at), device=p.device) - torch.repeat_interleave(torch.cumsum(count, 0) - count, count)
            nodes, cells = nodes[at], child[cells[at]] + within
    return torch.zeros_like(p).index_add(0, order, total)


def _simple(n, src, dst, w):
    src, dst = np.asarray(src, np.int64), np.asarray(dst, np.int64)
    lo, hi = np.minimum(src, dst), np.maximum(src, dst)
    at = np.nonzero(lo != hi)[0]
    _, first = np.unique(lo[at] * n + hi[at], return_index=True)
    at = at[np.sort(first)]
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    return t(lo[at]), t(hi[at]), t(np.ones(len(at)) if w is None else np.asarray(w, np.float64)[at]), at


def _fa2_tick(p, e, c, mass, gid, graphs, prm, ctl):
    """One ForceAtlas2 tick: positions after it and the controller after it. `prm`: each graph's values."""
    lo, hi = e
    at = lambda k: prm[k][gid]  # noqa: E731
    dist = lambda v: torch.sqrt((v * v).sum(1))  # noqa: E731

    def body(i, d, m):
        return d * (at("kr")[i] * mass[i] * m / (d * d).sum(1))[:, None]

    rep = _walk(p, mass, gid, graphs, lambda w2, d2, holds: ~holds & (w2 < prm["theta2"] * d2), body)
    d = p[hi] - p[lo]
    if prm["lin_log"]:
        r = dist(d)
        c = c * torch.log1p(r) / r
    att = torch.zeros_like(p).index_add(0, lo, d * c[:, None]).index_add(0, hi, -d * c[:, None])
    if prm["dissuade"]:
        att = att / mass[:, None]
    count = torch.bincount(gid, minlength=graphs).to(p.dtype)
    off = p - (_seg(gid, p, graphs) / count[:, None])[gid]
    pull = (at("gravity") * mass)[:, None]
    u = att + rep - (pull * off if prm["strong"] else pull * off / dist(off)[:, None])
    swing = ctl["swing"] + _seg(gid, mass * dist(p - u), graphs)
    traction = ctl["traction"] + _seg(gid, 0.5 * mass * dist(p + u), graphs)
    se, speed = ctl["se"], ctl["speed"]
    opt = 0.05 * torch.sqrt(count)
    jitter = torch.maximum(torch.sqrt(opt), torch.clamp(opt * traction / (count * count), max=10.0))
    rough = swing / traction > 2.0
    se = torch.where(rough & (se > 0.05), se * 0.5, se)
    jitter = torch.where(rough, torch.clamp(jitter, min=1.0), jitter)
    target = jitter * se * traction / swing
    much = swing > jitter * traction
    se = torch.where(much, torch.where(se > 0.05, se * 0.7, se), torch.where(speed < 1000.0, se * 1.3, se))
    speed = speed + torch.minimum(target - speed, 0.5 * speed)
    s = speed[gid]
    p = p + u * (s / (1.0 + torch.sqrt(s * mass * dist(u))))[:, None]
    return p, dict(swing=swing, traction=traction, se=se, speed=speed)


def _fa2_setup(n, src, dst, w, prms, gid, graphs):
    lo, hi, c, raw = _simple(n, src, dst, w)
    mass = 1.0 + torch.bincount(lo, minlength=n).double() + torch.bincount(hi, minlength=n).double()
    f = lambda k, d: torch.tensor([_f32(q.get(k, d)) for q in prms], dtype=torch.float64, device=DEV)  # noqa: E731
    prm = dict(kr=f("scaling_ratio", 2.0), gravity=f("gravity", 1.0), theta2=_f32(prms[0]["theta"] ** 2),
               lin_log=prms[0].get("lin_log", 0), dissuade=prms[0].get("dissuade_hubs", 0), strong=prms[0].get("strong_gravity", 0))
    one = torch.ones(graphs, dtype=torch.float64, device=DEV)
    return (lo, hi), c, raw, mass, prm, dict(swing=one, traction=one, se=one, speed=one)


def _fa2_exact(n, src, dst, w, pos, prms, ticks, gid=None, graphs=1):
    gid = torch.zeros(n, dtype=torch.long, device=DEV) if gid is None else gid
    e, c, _, mass, prm, ctl = _fa2_setup(n, src, dst, w, prms, gid, graphs)
    p, out = torch.from_numpy(pos).to(DEV).double(), []
    with torch.no_grad():
        for _ in range(ticks):
            p, ctl = _fa2_tick(p, e, c, mass, gid, graphs, prm, ctl)
            out.append(p)
    return out


def _mulberry(seed, count):
    a = (np.uint64(seed) + np.arange(1, count + 1, dtype=np.uint64) * np.uint64(0x6D2B79F5)) & np.uint64(0xFFFFFFFF)
    m = np.uint64(0xFFFFFFFF)
    t = (a ^ (a >> np.uint64(15))) * (a | np.uint64(1)) & m
    t = ((t + ((t ^ (t >> np.uint64(7))) * (t | np.uint64(61)) & m)) & m) ^ t
    return (t ^ (t >> np.uint64(14))).astype(np.float64) / 2.0 ** 32


def _near(p, reach):
    """Ordered pairs (i, j), i != j, of points closer than `reach`."""
    cell = (p / reach).floor().long()
    cell = cell - cell.amin(0) + 1
    wide = int(cell[:, 1].max()) + 2
    key = cell[:, 0] * wide + cell[:, 1]
    skey, order = torch.sort(key)
    ii, jj = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            want = key + dx * wide + dy
            a, b = torch.searchsorted(skey, want), torch.searchsorted(skey, want, right=True)
            count = b - a
            i = torch.repeat_interleave(torch.arange(len(p), device=p.device), count)
            j = order[torch.arange(len(i), device=p.device) - torch.repeat_interleave(torch.cumsum(count, 0) - count, count) + a[i]]
            keep = (i != j) & (((p[i] - p[j]) ** 2).sum(1) < reach * reach)
            ii.append(i[keep])
            jj.append(j[keep])
    return torch.cat(ii), torch.cat(jj)


def _mesh_field(p, dmin2, dmax):
    """The field of unit charges on the side x side mesh, read back at the points."""
    n = len(p)
    side = min(1024, max(128, 1 << max(0, math.ceil(math.log2(math.ceil(math.sqrt(n)))))))
    low, span = p.amin(0), float((p.amax(0) - p.amin(0)).max())
    step = max(-32, math.floor(4.0 * math.log2(span / side)))
    while True:
        h = 2.0 ** (step / 4.0)
        cells = math.floor(span / h) + 3
        reach = min(cells - 1, math.ceil(dmax / h))
        if cells <= side and cells + reach <= side:
            break
        step += 1
    u = (p - (low / h).floor() * h) / h
    c = u.floor().clamp(0, cells - 2)
    f = (u - c).clamp(0.0, 1.0)
    base = c[:, 1].long() * side + c[:, 0].long()
    corner = [(base + b * side + a, (f[:, 0] if a else 1 - f[:, 0]) * (f[:, 1] if b else 1 - f[:, 1])) for b in (0, 1) for a in (0, 1)]
    mesh = torch.zeros(side * side, dtype=torch.float64, device=p.device)
    for at, wt in corner:
        mesh.index_add_(0, at, wt)
    k = torch.arange(side, device=p.device)
    off = torch.where(k <= reach, k, torch.where(k >= side - reach, k - side, side * 4)).double()
    rx, ry = off[None, :] * h, off[:, None] * h
    r2 = rx * rx + ry * ry
    ok = (off[None, :] < side) & (off[:, None] < side) & (r2 > 0) & (r2 < dmax * dmax)
    l = torch.where(r2 < dmin2, torch.sqrt(dmin2 * r2), r2)
    green = torch.where(ok, 1.0 / l, torch.zeros_like(l))
    green = torch.complex(-rx * green, -ry * green)
    field = torch.fft.ifft2(torch.fft.fft2(mesh.view(side, side).to(torch.complex128)) * torch.fft.fft2(green)).reshape(-1)
    e = sum(torch.view_as_real(field[at]) * wt[:, None] for at, wt in corner)
    return e


def _force_exact(case, seed):
    n = case["n"]
    src, dst, st = _force_inputs(case, seed)
    lo, hi, s, _ = _simple(n, src, dst, st)
    s = s.float().double()
    deg = torch.bincount(lo, minlength=n).double() + torch.bincount(hi, minlength=n).double()
    i = np.arange(n, dtype=np.float64)
    radius, angle = 12.0 * np.sqrt(i + 1.0), i * 2.399963229728653
    p = torch.from_numpy(np.stack([np.cos(angle) * radius, np.sin(angle) * radius], 1).astype(np.float32)).to(DEV).double()
    v = torch.zeros_like(p)
    one, gid = torch.ones(n, dtype=torch.float64, device=DEV), torch.zeros(n, dtype=torch.long, device=DEV)
    alpha, theta2, dmax2, decay = 1.0, _f32(0.9 * 0.9), 520.0 ** 2, _f32(1.0 - 0.42)
    for _ in range(case["ticks"]):
        alpha += (0.0 - alpha) * 0.06
        pp = p + v
        d = pp[hi] - pp[lo]
        l = torch.sqrt((d * d).sum(1)).clamp(min=1e-300)
        f = d * ((l - 60.0 / s.clamp(min=0.4)) / l * alpha * (0.15 * s).clamp(max=0.7))[:, None]
        bias = (deg[lo] / (deg[lo] + deg[hi]))[:, None]
        v = v.index_add(0, hi, -f * bias).index_add(0, lo, f * (1 - bias))
        if case["mesh"]:
            v = v - 90.0 * alpha * _mesh_field(p, 1.0, 520.0)
        else:
            def body(k, d, m):
                l2 = (d * d).sum(1)
                g = torch.where(l2 < 1.0, torch.sqrt(l2), l2).clamp(min=1e-300)
                return d * (90.0 * alpha * torch.where(l2 < dmax2, m / g, torch.zeros_like(g)))[:, None]
            v = v + _walk(p, one, gid, 1, lambda w2, d2, holds: w2 < theta2 * d2, body)
        p = p - p.mean(0)
        pp = p + v
        a, b = _near(pp, 32.0)
        d = pp[a] - pp[b]
        l = torch.sqrt((d * d).sum(1)).clamp(min=1e-300)
        v = v.index_add(0, a, d * ((32.0 - l) / l * 0.5)[:, None])
        v = v * decay
        p = p + v
    return p, v


def _stress_exact(case, seed):
    n = case["n"]
    src, dst, x, y = _stress_inputs(case, seed)
    lo, hi, _, _ = _simple(n, src, dst, None)
    x, y = torch.from_numpy(x).to(DEV), torch.from_numpy(y).to(DEV)
    de = ee = dd = 0.0
    for v in range(0, n, max(n // 16, 1)):
        hop = torch.full((n,), -1, dtype=torch.long, device=DEV)
        hop[v] = 0
        for level in range(1, n):
            for a, b in ((lo, hi), (hi, lo)):
                to = b[hop[a] == level - 1]
                hop[to[hop[to] < 0]] = level
            if not (hop == level).any():
                break
        ok = hop > 0
        d, e = hop[ok].double(), torch.hypot((x[ok] - x[v]).double(), (y[ok] - y[v]).double())
        de, ee, dd = de + float((d * e).sum()), ee + float((e * e).sum()), dd + float((d * d).sum())
    return math.sqrt(max((dd - de / ee * de) / dd, 0.0))


def exact(case, seed):
    kind = case["kind"]
    if kind == "fa2":
        src, dst, w, pos = _fa2_inputs(case, seed)
        return torch.stack(_fa2_exact(case["n"], src, dst, w, pos, [_fa2_params(case, seed)], case["ticks"]))
    if kind == "call":
        src, dst, w = _graph(case["model"], case["n"], seed)
        prm = _fa2_params(case, seed)
        pos = _mulberry(prm["seed"], 2 * case["n"]).reshape(-1, 2).astype(np.float32)
        p = _fa2_exact(case["n"], src, dst, None, pos, [prm], case["ticks"])[-1]
        return p[:, 0], p[:, 1]
    if kind == "batch":
        gs = _batch_inputs(case, seed)
        off = np.cumsum([0] + [g.n for g in gs])
        src = np.concatenate([g.src.astype(np.int64) + o for g, o in zip(gs, off)])
        dst = np.concatenate([g.dst.astype(np.int64) + o for g, o in zip(gs, off)])
        gid = torch.repeat_interleave(torch.arange(len(gs)), torch.tensor([g.n for g in gs])).to(DEV)
        return _fa2_exact(int(off[-1]), src, dst, None, np.concatenate([g.pos0 for g in gs]), [g.params for g in gs], case["ticks"],
                          gid, len(gs))[-1]
    if kind == "backward":
        src, dst, w, pos, grad = _backward_inputs(case, seed)
        n = case["n"]
        gid = torch.zeros(n, dtype=torch.long, device=DEV)
        e, c, raw, mass, prm, ctl = _fa2_setup(n, src, dst, w, [dict(theta=case["theta"])], gid, 1)
        p = torch.from_numpy(pos).to(DEV).double().requires_grad_()
        c = c.float().double().requires_grad_()
        q, _ = _fa2_tick(p, e, c, mass, gid, 1, prm, ctl)
        dp, dc = torch.autograd.grad(q, [p, c], torch.from_numpy(grad).to(DEV).double())
        dw = torch.zeros(len(src), dtype=torch.float64, device=DEV)
        dw[torch.from_numpy(raw).to(DEV)] = dc
        return dp, dw
    if kind == "force":
        return _force_exact(case, seed)
    return _stress_exact(case, seed)
