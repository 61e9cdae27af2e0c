"""The layouts this engine is used for, as measurable cases.

A case is one pass of a program that lays graphs out: a few ForceAtlas2
iterations of a graph (or of a batch of graphs) and the positions back on the
host, the repulsion of bodies the caller holds on the device, or the picture
of a layout.  Graphs, positions, weights and sizes are drawn from the seed;
the sizes are those of the benchmark, the tests and the spans between them.

Kinds ("kind" of a case):

* layout   Engine.step_host with pinned host memory.  With "speed" 0, a program
           that keeps the positions itself: in, `iters` iterations, out; it
           comes back with the one and the other of two layouts in turn (the
           second a mirror image of the first, a little smaller, so the nodes
           swing and the speed rule stays away from its thresholds).
           With "speed" above 0, a layout resumed at that global speed (a
           running layout's is small) that goes on from pass to pass:
           `iters` iterations, positions out.
* batch    BatchEngine: positions in, `iters` iterations of every graph,
           positions out, two layouts in turn.
* noalloc  fa2_repulsion_noalloc on device tensors (the C ABI's entry point
           for callers that may not allocate).
* render   render_rgb: the picture the command line writes of a layout.
"""
import ctypes
import math

import numpy as np
import torch

from gpugraphlayout_b200 import BatchEngine, Engine, FarFieldMLP, _native, render_rgb

EPS = 0.05 * 0.05
SPEED = 1e-6  # global speed a resumed layout starts at


def _layout(name=None, **kw):
    """A layout case: plain values only; options left out are off."""
    c = {"kind": "layout", "graph": "ba", "n": 1000, "m": 3, "strong": True, "scale": 10.0,
         "gravity": 1.0, "width": 20000.0, "theta": 1.0, "multipole": 1, "linlog": False,
         "delta": 0.0, "overlap": False, "learned": False, "speed": 0.0, "iters": 1}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest use: an interactive view of a few hundred nodes, where
        # the launches and the waits of an iteration are all there is
        _layout("small_view", graph="ba", n=300, m=2, strong=False, scale=80.0, width=2000.0,
                speed=SPEED, iters=4),
        # the configuration the reference's CPU path is quoted on, running
        _layout("ba10k", graph="ba", n=10000, m=3, strong=False, scale=80.0, width=10000.0,
                speed=SPEED, iters=4),
        # one iteration with the positions in from and out to the host, as a
        # program that keeps its own layout calls it
        _layout("rmat16_host", graph="rmat", n=46717, m=22),
        # the headline workload, end to end
        _layout("rmat20", graph="rmat", n=646567, m=26),
        # the quadrupole walk at the opening angle that gives the plain
        # walk's error
        _layout("rmat18_quadrupole", graph="rmat", n=163839, m=20, theta=1.7, multipole=2,
                speed=SPEED, iters=3),
        # weighted communities with linear-log attraction
        _layout("sbm100k_weighted_linlog", graph="sbm", n=100003, m=10, strong=False, scale=2.0,
                linlog=True, delta=0.7),
        # node sizes that must not overlap
        _layout("ba30k_overlap", graph="ba", n=30011, m=4, strong=False, scale=10.0,
                overlap=True),
        # the learned far-field correction at its working opening angle
        _layout("rmat17_learned", graph="rmat", n=90210, m=22, theta=1.6, learned=True),
        # many small graphs side by side (a gallery of communities)
        {"name": "batch_small", "kind": "batch", "graphs": 96, "n_min": 50, "n_max": 600,
         "iters": 1},
        # the batched workload: 50 to 20,000 nodes a graph
        {"name": "batch_wide", "kind": "batch", "graphs": 512, "n_min": 50, "n_max": 20000,
         "iters": 1},
        # a caller's own bodies on the device
        {"name": "noalloc_5003", "kind": "noalloc", "n": 5003, "scale": 10.0, "theta": 1.0},
        # the command line's picture
        {"name": "render_1250", "kind": "render", "n": 46000, "m": 8, "width": 1250,
         "height": 1250},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.random()
    if k < 0.15:
        lo = rng.randint(2, 400)
        graphs = _log(rng, 8, 400)
        return {"kind": "batch", "graphs": graphs, "n_min": lo,
                "n_max": _log(rng, lo + 1, 20000), "iters": 1}
    if k < 0.25:
        return {"kind": "noalloc", "n": _log(rng, 2, 8192),
                "scale": round(rng.uniform(1.0, 80.0), 2),
                "theta": round(rng.uniform(0.5, 1.5), 2)}
    if k < 0.32:
        return {"kind": "render", "n": _log(rng, 10, 100000), "m": rng.randint(1, 8),
                "width": rng.randint(200, 2000), "height": rng.randint(200, 2000)}
    graph = rng.choice(["ba", "rmat", "sbm"])
    c = _layout(graph=graph, n=_log(rng, 33, 600000), m=rng.randint(2, 16),
                strong=rng.random() < 0.5, scale=round(rng.uniform(1.0, 80.0), 2),
                gravity=round(rng.uniform(0.5, 2.0), 2),
                width=round(math.exp(rng.uniform(math.log(1e3), math.log(2e4))), 1),
                speed=0.0)
    if graph != "rmat" and c["n"] <= 50000 and rng.random() < 0.7:
        c.update(speed=SPEED, iters=rng.randint(1, 4))
    o = rng.random()
    if o < 0.2:
        c.update(multipole=2, theta=round(rng.uniform(1.0, 2.0), 2))
    elif o < 0.35:
        c.update(linlog=True)
    elif o < 0.5:
        c.update(delta=round(rng.uniform(0.3, 1.5), 2), linlog=rng.random() < 0.5)
    elif o < 0.6:
        c.update(overlap=True, speed=0.0, iters=1)
    elif o < 0.7 and c["n"] > 2000:
        c.update(learned=True, theta=round(rng.uniform(1.2, 2.0), 2), speed=0.0, iters=1)
    elif o < 0.85:
        c.update(theta=round(rng.uniform(0.6, 1.5), 2))
    return c


# ------------------------------------------------------------------ inputs --


def _dedupe(n, s, t):
    """Undirected edges once each as (lo, hi), self-loops dropped."""
    lo, hi = torch.minimum(s, t), torch.maximum(s, t)
    key = torch.unique((lo * n + hi)[lo != hi])
    return key // n, key % n


def _rmat(n, m, g):
    """R-MAT (a, b, c, d) = (.57, .19, .19, .05), n m draws over the power of
    two ids of which about n get an edge; those packed to n nodes (the few
    past n dropped, the few missing tied to the first nodes)."""
    scale = max(1, int(1.4 * n).bit_length())
    draws = n * m
    s = torch.zeros(draws, dtype=torch.int64, device="cuda")
    t = torch.zeros(draws, dtype=torch.int64, device="cuda")
    for lvl in range(scale):
        r = torch.rand(draws, generator=g, device="cuda")
        s |= (r >= 0.76).long() << lvl
        t |= (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long() << lvl
    s, t = _dedupe(1 << scale, s, t)
    inv = torch.unique(torch.cat([s, t]), return_inverse=True)[1]
    k = int(inv.max()) + 1
    e = inv.reshape(2, -1)
    e = e[:, (e < n).all(0)]
    late = torch.arange(min(k, n), n, device="cuda")
    return torch.cat([e[0], late % max(1, min(k, n) - 1)]), torch.cat([e[1], late])


def _ba(n, m, g):
    """Preferential attachment: node v's j-th edge ends where a uniformly
    drawn earlier end of an edge does (Batagelj and Brandes 2005), all nodes
    at once by pointer doubling."""
    k = n * m
    node = torch.arange(k, device="cuda") // m
    src = 2 * torch.arange(k, device="cuda")
    ptr = torch.arange(2 * k, device="cuda")
    r = (torch.rand(k, generator=g, device="cuda", dtype=torch.float64) * (src + 1)).long()
    ptr[src + 1] = torch.minimum(r, src)
    for _ in range(2 * k.bit_length()):
        nxt = ptr[ptr]
        if torch.equal(nxt, ptr):
            break
        ptr = nxt
    return _dedupe(n, node, node[ptr[src + 1] // 2])


def _sbm(sizes, degree, g):
    """Communities, one stochastic block model per entry of `sizes`: a tenth
    of the edges between blocks.  Returns node offsets and edges over all."""
    sizes = torch.as_tensor(sizes, device="cuda", dtype=torch.int64)
    off = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), sizes.cumsum(0)])
    n = int(off[-1])
    which = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), sizes)
    block = (sizes // 16).clamp(min=2)[which]
    base = off[which]
    node = torch.arange(n, device="cuda") - base
    per = max(1, degree // 2)
    node, block, base, sz = (x.repeat_interleave(per) for x in (node, block, base, sizes[which]))
    u = torch.rand(len(node), generator=g, device="cuda", dtype=torch.float64)
    inner = torch.rand(len(node), generator=g, device="cuda") < 0.9
    b0 = node // block * block
    width = torch.minimum(block, sz - b0)
    other = torch.where(inner, b0 + (u * width).long(), (u * sz).long())
    lo, hi = torch.minimum(node, other) + base, torch.maximum(node, other) + base
    key = torch.unique((lo * n + hi)[lo != hi])
    return off, key // n, key % n


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _graph(case, seed):
    g = _gen(seed)
    if case["graph"] == "rmat":
        s, t = _rmat(case["n"], case["m"], g)
    elif case["graph"] == "ba":
        s, t = _ba(case["n"], case["m"], g)
    else:
        _, s, t = _sbm([case["n"]], 2 * case["m"], g)
    return g, case["n"], s, t


def _layout_inputs(case, seed):
    g, n, s, t = _graph(case, seed)
    if case["speed"]:  # a running layout: dense in the middle
        r = torch.rand(n, 1, generator=g, device="cuda").pow(0.75) * (0.5 * case["width"])
        a = torch.rand(n, 1, generator=g, device="cuda") * (2 * math.pi)
        xy = torch.cat([r * a.cos(), r * a.sin()], 1)
    else:  # a fresh one, as randomizePositions draws it
        xy = (torch.rand(n, 2, generator=g, device="cuda") - 0.5) * case["width"]
    w = (0.1 + 3.0 * torch.rand(s.numel(), generator=g, device="cuda")) if case["delta"] else None
    # sizes of up to a third of the mean spacing of the start
    size = None
    if case["overlap"]:
        size = torch.rand(n, generator=g, device="cuda") * (case["width"] / math.sqrt(n) / 3)
    return n, s, t, xy, w, size


def _mlp(seed):
    """A model whose corrections have the size of a trained one's (a few
    percent of the cell's own term)."""
    mlp = FarFieldMLP(seed=int(seed) & 0xFFFF)
    mlp["w3"] = mlp["w3"] * 0.05
    mlp["b3"] = mlp["b3"] * 0.0
    return mlp


def _batch_inputs(case, seed):
    g = _gen(seed)
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    u = (torch.arange(case["graphs"], dtype=torch.float64, device="cuda") + 0.5) / case["graphs"]
    sizes = torch.exp(lo + u * (hi - lo)).round().long()
    off, s, t = _sbm(sizes, 32, g)
    n = int(off[-1])
    which = torch.repeat_interleave(torch.arange(case["graphs"], device="cuda"), sizes)
    xy = (torch.rand(n, 2, generator=g, device="cuda") - 0.5) * (20.0 * sizes[which, None].float().sqrt())
    return off, which, s, t, xy


def _u32(x):
    return x.to(torch.int32).cpu().numpy().view(np.uint32)


def _pinned(xy):
    return torch.empty((len(xy), 2), dtype=torch.float32, pin_memory=True).copy_(xy)


def prepare(case, seed):
    if case["kind"] == "layout":
        n, s, t, xy, w, size = _layout_inputs(case, seed)
        e = Engine(n, _u32(s), _u32(t), strong_gravity=case["strong"], gravity=case["gravity"],
                   scale=case["scale"], theta=case["theta"], multipole=case["multipole"],
                   linlog=case["linlog"], weights=None if w is None else w.cpu().numpy(),
                   delta=case["delta"])
        host = _pinned(xy)
        e.set_positions(host.numpy())
        if case["speed"]:
            e.set_speed_state(case["speed"], 1.0)
        if size is not None:
            e.set_prevent_overlap(size.cpu().numpy())
        if case["learned"]:
            e.set_learned_correction(_mlp(seed))
        return {"case": case, "engine": e, "out": host, "turn": 0,
                "xy": [_pinned(xy), _pinned(-0.8 * xy)]}
    if case["kind"] == "batch":
        off, _, s, t, xy = _batch_inputs(case, seed)
        off = off.cpu().numpy()
        sh, th = s.cpu().numpy(), t.cpu().numpy()
        cut = np.searchsorted(sh, off)
        graphs = [(int(off[i + 1] - off[i]), (sh[cut[i]:cut[i + 1]] - off[i]).astype(np.uint32),
                   (th[cut[i]:cut[i + 1]] - off[i]).astype(np.uint32))
                  for i in range(len(off) - 1)]
        b = BatchEngine(graphs, strong_gravity=False, gravity=1.0, scale=2.0)
        # the class split the autotuner picks on this mix
        b.configure(4096, 512, 1024)
        return {"case": case, "engine": b, "out": _pinned(xy), "turn": 0,
                "xy": [_pinned(xy), _pinned(-0.8 * xy)]}
    g = _gen(seed)
    if case["kind"] == "noalloc":
        n = case["n"]
        xy = torch.randn(n, 2, generator=g, device="cuda") * 500.0
        mass = (1.0 + torch.rand(n, generator=g, device="cuda").pow(-0.7).clamp(max=500.0)).floor()
        prm = _native.Params()
        _native.lib().fa2_default_params(ctypes.byref(prm))
        prm.scale, prm.theta = case["scale"], case["theta"]
        return {"case": case, "xy": xy, "mass": mass, "prm": prm, "out": torch.empty_like(xy)}
    n = case["n"]
    s, t = _ba(n, case["m"], g)
    # a relaxed layout's shape: dense centre, half the nodes near a neighbour
    xy = torch.randn(n, 2, generator=g, device="cuda") * 1000.0
    first = torch.full((n,), n, device="cuda").scatter_reduce(0, t, s, "amin")
    near = (torch.rand(n, generator=g, device="cuda") < 0.5) & (first < n)
    xy[near] = xy[first[near]] + 50.0 * torch.randn(int(near.sum()), 2, generator=g, device="cuda")
    return {"case": case, "n": n, "src": _u32(s), "dst": _u32(t), "xy": xy.cpu().numpy()}


# --------------------------------------------------------------------- run --


def run(state):
    case = state["case"]
    if case["kind"] in ("layout", "batch"):
        e, out = state["engine"], state["out"]
        xy = state["xy"][state["turn"]]
        state["turn"] ^= 1
        if case["kind"] == "layout":
            e.step_host(None if case["speed"] else xy.data_ptr(), case["iters"], out.data_ptr())
        else:
            e.set_positions_ptr(xy.data_ptr())
            e.step(case["iters"])
            e.get_positions_ptr(out.data_ptr())
        return out
    if case["kind"] == "noalloc":
        _native.check(_native.lib().fa2_repulsion_noalloc(
            ctypes.c_void_p(state["xy"].data_ptr()), ctypes.c_void_p(state["mass"].data_ptr()),
            case["n"], ctypes.byref(state["prm"]),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
            ctypes.c_void_p(state["out"].data_ptr())), "fa2_repulsion_noalloc")
        return state["out"]
    return render_rgb(state["n"], state["src"], state["dst"], state["xy"], case["width"],
                      case["height"])


def work(case):
    """Bytes: the edges' two directions, positions, forces and masses of each
    iteration once, and the positions over the bus.  FLOPs: 10 per body-node
    term of the walk, about 22 log2(n) / theta^2 terms per body (456 at
    n = 646,567, theta 1)."""
    if case["kind"] == "layout":
        n, e = case["n"], case["n"] * case["m"]
        it = case["iters"]
        flops = it * 10.0 * 22.0 * math.log2(n + 1) / case["theta"] ** 2 * n
        if case["multipole"] == 2:
            flops *= 2.4
        return {"bytes": it * ((8 + 8 * bool(case["delta"])) * e + 64.0 * n) +
                8.0 * n * (1 if case["speed"] else 2), "flops": flops}
    if case["kind"] == "batch":
        lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
        n = case["graphs"] * ((math.exp(hi) - math.exp(lo)) / (hi - lo) if hi > lo else case["n_min"])
        mid = math.exp(0.5 * (lo + hi))
        return {"bytes": case["iters"] * (8.0 * 15 * n + 64.0 * n) + 16.0 * n,
                "flops": case["iters"] * 220.0 * math.log2(mid + 2) * n}
    if case["kind"] == "noalloc":
        n = case["n"]
        return {"bytes": 20.0 * n, "flops": 220.0 * math.log2(n + 1) / case["theta"] ** 2 * n}
    pixels = case["width"] * case["height"]
    return {"bytes": 8.0 * case["n"] * (1 + case["m"]) + 3.0 * pixels,
            "flops": 10.0 * pixels}


# ------------------------------------------------------------------- exact --


def _repulsion(xy, mass, k_r, size=None):
    """k_r m_i sum_j m_j d / (d^2 + eps) over all pairs (with sizes, the
    anti-collision rule on the border-to-border distance)."""
    n = len(xy)
    out = torch.zeros_like(xy)
    step = max(1, (1 << 26) // n)
    for a in range(0, n, step):
        b = min(n, a + step)
        dx = xy[a:b, None, 0] - xy[None, :, 0]
        dy = xy[a:b, None, 1] - xy[None, :, 1]
        d2 = dx * dx + dy * dy + EPS
        if size is None:
            c = mass / d2
        else:
            d = d2.sqrt()
            gap = d - size[a:b, None] - size[None, :]
            c = torch.where(gap > 0, mass / (d * gap), torch.where(gap < 0, 100 * mass / d, 0.0))
        out[a:b, 0] = (dx * c).sum(1)
        out[a:b, 1] = (dy * c).sum(1)
    return out * (k_r * mass)[:, None]


def _iterate(xy, s, t, case, w=None, size=None):
    """`iters` ForceAtlas2 iterations in float64 with the direct sum."""
    n = len(xy)
    one = torch.ones(len(s), dtype=torch.float64, device=xy.device)
    mass = torch.ones(n, dtype=torch.float64, device=xy.device)
    mass.index_add_(0, s, one)
    mass.index_add_(0, t, one)
    fprev = torch.zeros_like(xy)
    gs, se = case["speed"] or 1.0, 1.0
    pull = one if w is None else w
    for _ in range(case["iters"]):
        d = xy[t] - xy[s]
        dist = d.norm(dim=1)
        f = pull[:, None] * d
        if case["linlog"]:
            f = f * torch.where(dist > 0, torch.log1p(dist) / dist, 0.0)[:, None]
        if size is not None:
            gap = dist - size[s] - size[t]
            f = f * torch.where(gap > 0, gap / dist, 0.0)[:, None]
        r = xy.norm(dim=1)
        g = case["gravity"] * mass
        if not case["strong"]:
            g = torch.where(r > 0, g / r, 0.0)
        tot = -g[:, None] * xy
        tot.index_add_(0, s, f)
        tot.index_add_(0, t, -f)
        tot = tot + _repulsion(xy, mass, case["scale"], size)
        swing = float((mass * (tot - fprev).norm(dim=1)).sum())
        tra = float((mass * (tot + fprev).norm(dim=1) / 2).sum())
        opt = 0.05 * math.sqrt(n)
        jt = max(math.sqrt(opt), min(10.0, opt * tra / n ** 2))
        if swing / tra > 2.0 + 1e-9:
            if se > 0.05:
                se *= 0.5
            jt = max(jt, 1.0)
        target = jt * se * tra / swing
        if swing > jt * tra:
            if se > 0.05:
                se *= 0.7
        elif gs < 1000:
            se *= 1.3
        gs += min(target - gs, 0.5 * gs)
        xy = xy + tot * (gs / (1 + (gs * (tot - fprev).norm(dim=1)).sqrt()))[:, None]
        fprev = tot
    return xy


def exact(case, seed):
    if case["kind"] == "layout":
        if case["n"] ** 2 * case["iters"] > 2e11:
            return None
        n, s, t, xy, w, size = _layout_inputs(case, seed)
        w = None if w is None else w.double() ** case["delta"]
        return _iterate(xy.double(), s, t, case, w, None if size is None else size.double())
    if case["kind"] == "batch":
        off, which, s, t, xy = _batch_inputs(case, seed)
        c = dict(case, strong=False, gravity=1.0, scale=2.0, linlog=False, speed=0.0)
        off, xy = off.tolist(), xy.double()
        cut = torch.searchsorted(s, torch.tensor(off, device="cuda")).tolist()
        out = [_iterate(xy[a:b], s[p:q] - a, t[p:q] - a, c)
               for a, b, p, q in zip(off, off[1:], cut, cut[1:])]
        return torch.cat(out)
    if case["kind"] == "noalloc":
        st = prepare(case, seed)
        return _repulsion(st["xy"].double(), st["mass"].double(), case["scale"])
    return None
