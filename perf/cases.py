"""Workloads for timing the engine through its public entry points.

A case is a dict of plain values. ``listed()`` gives the standing cases,
``draw(rng)`` another one of the same ranges, ``prepare(case, seed)`` what a
program holds before the call, ``run(state)`` one pass, ``work(case)`` the
bytes and operations a pass cannot do without and ``exact(case, seed)`` the
computed numbers in 64 bits by plain torch.

Polygons are the benchmark's seeded stars: centres uniform in a square, mean
radius and vertex count log-uniform, vertex angles sorted uniform, per-vertex
radius x lognormal(0, 0.3). They are drawn on the GPU, so that large inputs
are quick to make.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from farm_gb300.engine import MODE_APPROX, MODE_EXACT, Store

SIGMA = 0.3
IN, IN_PAD, HID = 520, 576, 256  # the scorer's features, their padding, its hidden width


def listed() -> list:
    return [
        # a handful of candidate pairs asked of a store that is already
        # rasterized: an interactive lookup, all latency
        {"name": "query_few", "kind": "query", "ns": 40, "nt": 120, "n_lo": 16, "n_hi": 600, "side": 12.0, "vpr": 10,
         "cc": 16, "pairs": 48, "mode": MODE_EXACT, "device": False},
        # two small files joined from host memory: load, rasterize, candidates, intersect
        {"name": "join_few", "kind": "join", "ns": 40, "nt": 120, "n_lo": 16, "n_hi": 600, "side": 12.0, "vpr": 10,
         "cc": 16, "device": False},
        # the ordinary join (configuration 1): 1,000 x 10,000 polygons of up to 1,024 vertices, -v 10, host arrays
        {"name": "join_ordinary", "kind": "join", "ns": 1000, "nt": 10000, "n_lo": 16, "n_hi": 1024, "side": 100.0,
         "vpr": 10, "cc": 16, "device": False},
        # a piece of the heavy-tailed join (configuration 2) at the benchmark's -v 64: polygons of up to 100,000
        # vertices, rings resident on the device
        {"name": "join_heavy", "kind": "join", "ns": 301, "nt": 2999, "n_lo": 16, "n_hi": 100000, "side": 21.0,
         "vpr": 64, "cc": 16, "device": True},
        # a large candidate list on a standing store at -v 128 and 8-bit fill classes, device pairs
        {"name": "query_many", "kind": "query", "ns": 1001, "nt": 3003, "n_lo": 16, "n_hi": 20000, "side": 15.0,
         "vpr": 128, "cc": 256, "pairs": 150001, "mode": MODE_EXACT, "device": True},
        # containment report on a standing store: a million (polygon, point) pairs and the polygon pairs
        {"name": "contain_many", "kind": "contain", "ns": 1500, "nt": 2500, "n_lo": 16, "n_hi": 5000, "side": 15.0,
         "vpr": 10, "cc": 16, "pairs": 40001, "points": 1000003},
        # within 10 km in degrees, self-join, the whole path from host arrays with the hierarchical rasters
        {"name": "within_geo", "kind": "within_join", "n": 403, "n_lo": 16, "n_hi": 1500, "side": 25.0, "vpr": 10,
         "cc": 16},
        # within 10 km on projected coordinates in km (a cut of configuration 3), a standing store, device pairs
        {"name": "within_planar", "kind": "within_query", "n": 1001, "n_lo": 32, "n_hi": 20000, "side": 354.0,
         "vpr": 10, "cc": 16, "pairs": 60001},
        # overlap areas of two small layers from host arrays: load, rasterize, areas (the first call after a
        # rasterization builds the area's own indexes)
        {"name": "area_join", "kind": "area_join", "ns": 203, "nt": 405, "n_lo": 8, "n_hi": 1024, "side": 20.0,
         "vpr": 10, "cc": 16, "pairs": 1501},
        # a batch of mixed tiny and huge pairs through a captured area plan (a cut of configuration 4)
        {"name": "area_batch", "kind": "area_plan", "ns": 301, "nt": 299, "n_lo": 8, "n_hi": 20000, "side": 18.0,
         "vpr": 10, "cc": 16, "pairs": 801},
        # the learned scorer's probabilities of a long candidate list
        {"name": "score_many", "kind": "score", "ns": 1001, "nt": 3003, "n_lo": 16, "n_hi": 2000, "side": 13.0,
         "vpr": 64, "cc": 16, "pairs": 200003},
        # one training batch of the scorer, forward and backward (the trainer's batch size)
        {"name": "score_grad", "kind": "grad", "rows": 4096},
    ]


def _log(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    """One more case of the listed ones' ranges: the kind, then its sizes and options."""
    kind = rng.choice(["query", "join", "contain", "within_join", "within_query", "area_join", "area_plan", "score",
                       "grad"])
    if kind == "grad":
        return {"kind": kind, "rows": int(_log(rng, 100, 4096))}
    vpr = rng.choice([10, 10, 64, 128])
    cc = rng.choice([4, 16, 16, 256])
    if kind == "within_join":
        n = int(_log(rng, 50, 403))
        return {"kind": kind, "n": n, "n_lo": 16, "n_hi": int(_log(rng, 200, 1500)),
                "side": 25.0 * math.sqrt(n / 403), "vpr": rng.choice([10, 64]), "cc": cc}
    if kind == "within_query":
        n = int(_log(rng, 50, 1001))
        return {"kind": kind, "n": n, "n_lo": 32, "n_hi": int(_log(rng, 1000, 20000)),
                "side": 354.0 * math.sqrt(n / 1001), "vpr": 10, "cc": cc, "pairs": int(_log(rng, 100, 60 * n))}
    top = {"query": 20000, "join": 100000, "contain": 5000, "area_join": 1024, "area_plan": 20000, "score": 2000}
    low = {"query": 600, "join": 600, "contain": 600, "area_join": 200, "area_plan": 1000, "score": 600}
    most = {"query": 4004, "join": 11000, "contain": 4000, "area_join": 608, "area_plan": 600, "score": 4004}
    n_hi = int(_log(rng, low[kind], top[kind]))
    n = int(_log(rng, 160, most[kind]))
    if kind == "join":  # no more vertices than join_heavy, no more polygons than join_ordinary
        n = min(n, int(3300 * _mean_nv(16, 100000) / _mean_nv(16, n_hi)))
    ns = max(20, int(n * rng.uniform(0.1, 0.5)))
    case = {"kind": kind, "ns": ns, "nt": max(20, n - ns), "n_lo": 16, "n_hi": n_hi, "vpr": vpr, "cc": cc}
    # the side at which the boxes of the two sets give some pairs per polygon, as in the listed cases
    case["side"] = math.sqrt(15.0 * case["ns"] * case["nt"] / (n * rng.uniform(3.0, 10.0)))
    if kind == "query":
        case["pairs"] = int(_log(rng, 48, 10 * n))
        case["mode"] = rng.choice([MODE_EXACT, MODE_EXACT, MODE_EXACT, MODE_APPROX])
        case["device"] = rng.random() < 0.5
    elif kind == "join":
        case["device"] = rng.random() < 0.5
    elif kind == "contain":
        case["pairs"] = int(_log(rng, 100, 10 * n))
        case["points"] = int(_log(rng, 1000, 1000003))
    elif kind in ("area_join", "area_plan"):
        case["n_lo"] = 8
        case["vpr"] = rng.choice([10, 64])
        case["pairs"] = int(_log(rng, 100, 1501 if kind == "area_join" else 801))
    else:
        case["pairs"] = int(_log(rng, 100, 200003))
    return case


# ------------------------------------------------------------------ inputs --
def _mean_nv(lo: float, hi: float) -> float:
    return (hi - lo) / math.log(hi / lo)


def _stars(gen, n: int, n_lo: int, n_hi: int, r_lo: float, r_hi: float, side: float):
    """n star polygons on the GPU: offsets int64 [n + 1] and float32 vertices
    [total, 2], each ring closed by a copy of its first vertex."""
    dev = torch.device("cuda")

    def uni(*shape):
        return torch.rand(shape, generator=gen, device=dev, dtype=torch.float64)

    cnt = torch.exp(math.log(n_lo) + uni(n) * math.log(n_hi / n_lo)).long().clamp_(n_lo, n_hi)
    c = uni(n, 2) * side
    rbar = torch.exp(math.log(r_lo) + uni(n) * math.log(r_hi / r_lo))
    off = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    off[1:] = torch.cumsum(cnt + 1, 0)
    pid = torch.repeat_interleave(torch.arange(n, device=dev), cnt)
    ang = torch.sort(pid.double() + uni(len(pid))).values - pid.double()
    ang = ang.clamp_(0.0, 1.0) * (2.0 * math.pi)
    z = torch.randn(len(pid), generator=gen, device=dev, dtype=torch.float64)
    r = rbar[pid] * torch.exp(SIGMA * z)
    xy = torch.empty((int(off[-1]), 2), dtype=torch.float32, device=dev)
    at = torch.arange(len(pid), device=dev) + pid
    xy[at, 0] = (c[pid, 0] + r * torch.cos(ang)).float()
    xy[at, 1] = (c[pid, 1] + r * torch.sin(ang)).float()
    xy[off[1:] - 1] = xy[off[:-1]]
    return off, xy


def _boxes(off, xy):
    n = len(off) - 1
    pid = torch.repeat_interleave(torch.arange(n, device=xy.device), off[1:] - off[:-1])
    out = torch.empty((n, 4), dtype=torch.float32, device=xy.device)
    for k in range(2):
        out[:, k] = torch.full((n,), math.inf, device=xy.device).scatter_reduce(0, pid, xy[:, k], "amin")
        out[:, 2 + k] = torch.full((n,), -math.inf, device=xy.device).scatter_reduce(0, pid, xy[:, k], "amax")
    return out


def _pairs(gen, bs, bt, most: int, expand: float = 0.0, skip_same: bool = False):
    """`most` pairs (int32 [most, 2]) whose boxes overlap, at random and sorted; a
    list shorter than that is asked again."""
    e = expand
    hit = ((bs[:, None, 0] <= bt[None, :, 2] + e) & (bt[None, :, 0] <= bs[:, None, 2] + e) &
           (bs[:, None, 1] <= bt[None, :, 3] + e) & (bt[None, :, 1] <= bs[:, None, 3] + e))
    if skip_same:
        hit.fill_diagonal_(False)
    flat = torch.nonzero(hit.flatten()).flatten()
    perm = torch.randperm(len(flat), generator=gen, device=flat.device)
    flat = torch.sort(flat[perm[torch.arange(most, device=flat.device) % len(flat)]]).values
    return torch.stack([flat // len(bt), flat % len(bt)], 1).to(torch.int32).contiguous()


def _results(case: dict, n_s: int, n_t: int, device: bool):
    """A program's result buffers of a join: room for the candidates and a flag
    each, several times the expected number (255 and zeros past the last)."""
    cap = min(n_s * n_t, int(40.0 * n_s * n_t / case["side"] ** 2) + 2000)
    if device:
        return torch.zeros((cap, 2), dtype=torch.int32, device="cuda"), \
            torch.full((cap,), 255, dtype=torch.uint8, device="cuda")
    return np.zeros((cap, 2), np.uint32), np.full(cap, 255, np.uint8)


def _host(off, xy):
    return off.cpu().numpy().view(np.uint64), np.ascontiguousarray(xy.cpu().numpy())


def _host_pairs(p):
    return np.ascontiguousarray(p.cpu().numpy().view(np.uint32))


def _two_sets(case: dict, gen):
    r_lo = 0.3 if case["kind"] in ("area_join", "area_plan") else 0.05  # rings whose float32 vertices stay simple
    a = _stars(gen, case["ns"], case["n_lo"], case["n_hi"], r_lo, 2.0, case["side"])
    b = _stars(gen, case["nt"], case["n_lo"], case["n_hi"], r_lo, 2.0, case["side"])
    return a, b


def _generator(seed: int):
    return torch.Generator(device="cuda").manual_seed(seed)


def _grad_inputs(case: dict, seed: int):
    """Weights, features and labels of one batch: two 16 x 16 fill grids per row
    (discs of random centre and radius, in 15ths as 4-bit fills are) and eight
    size features; a row is positive where the discs meet."""
    gen = _generator(seed)
    dev = torch.device("cuda")

    def uni(*shape):
        return torch.rand(shape, generator=gen, device=dev, dtype=torch.float64)

    n = case["rows"]
    rows = (n + 127) // 128 * 128
    par = torch.empty(HID * IN_PAD + HID * HID + 3 * HID + 1, dtype=torch.float64, device=dev)
    o = 0
    for size, a in ((HID * IN_PAD, math.sqrt(6.0 / (IN + HID))), (HID * HID, math.sqrt(6.0 / (2 * HID))), (HID, 0.05),
                    (HID, 0.05), (HID, math.sqrt(6.0 / (HID + 1))), (1, 0.05)):
        par[o:o + size] = a * (2.0 * uni(size) - 1.0)
        o += size
    g = (torch.arange(16, device=dev, dtype=torch.float64) + 0.5) / 16.0
    gy, gx = torch.meshgrid(g, g, indexing="ij")
    c, r = uni(2, n, 2), 0.1 + 0.6 * uni(2, n)
    x = torch.zeros((rows, IN_PAD), dtype=torch.float64, device=dev)
    for k in range(2):
        d = torch.sqrt((gx[None] - c[k, :, 0, None, None]) ** 2 + (gy[None] - c[k, :, 1, None, None]) ** 2)
        fill = (0.5 + 8.0 * (r[k][:, None, None] - d)).clamp(0.0, 1.0)
        x[:n, 256 * k:256 * k + 256] = (torch.round(fill * 15.0) / 15.0).reshape(n, 256)
    x[:n, 512:520] = uni(n, 8) * 2.0 - 1.0
    y = torch.zeros(rows, dtype=torch.uint8, device=dev)
    y[:n] = (torch.sqrt(((c[0] - c[1]) ** 2).sum(1)) < r[0] + r[1] - 0.3).to(torch.uint8)
    return par.float(), x.to(torch.bfloat16).contiguous(), y


# --------------------------------------------------------------- the passes --
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = Store()
    state = {"kind": kind, "store": st}
    if kind == "grad":
        par, x, y = _grad_inputs(case, seed)
        st.mlp_load(par.cpu().numpy())
        state.update(x=x, y=y, n=case["rows"])
        return state
    gen = _generator(seed)
    opts = {"vpr": case["vpr"], "category_count": case["cc"], "strict": False}
    state["opts"] = opts
    if kind in ("within_join", "within_query"):
        r_lo, r_hi = (0.05, 2.0) if kind == "within_join" else (0.05, 50.0)
        off, xy = _stars(gen, case["n"], case["n_lo"], case["n_hi"], r_lo, r_hi, case["side"])
        opts["hierarchy"] = True
        if kind == "within_join":
            state["source"] = _host(off, xy)
            state["cand"], state["flags"] = _results(case, case["n"], case["n"], False)
        else:
            b = _boxes(off, xy)
            st.load(0, off, xy)
            st.rasterize(**opts)
            state["pairs"] = _pairs(gen, b, b, case["pairs"], expand=10.0, skip_same=True)
        torch.cuda.synchronize()
        return state
    a, b = _two_sets(case, gen)
    if kind == "join":
        state["device"] = case["device"]
        state["source"], state["target"] = (a, b) if case["device"] else (_host(*a), _host(*b))
        state["cand"], state["flags"] = _results(case, case["ns"], case["nt"], case["device"])
        torch.cuda.synchronize()
        return state
    ba, bb = _boxes(*a), _boxes(*b)
    pairs = _pairs(gen, ba, bb, case["pairs"])
    torch.cuda.synchronize()
    if kind == "area_join":
        state.update(source=_host(*a), target=_host(*b), pairs=_host_pairs(pairs))
        return state
    st.load(0, *a)
    st.load(1, *b)
    st.rasterize(**opts)
    state["pairs"] = pairs
    if kind == "query":
        state["mode"] = case["mode"]
        if not case["device"]:
            state["pairs"] = _host_pairs(pairs)
    elif kind == "contain":
        n = case["points"]
        poly = torch.randint(case["ns"], (n,), generator=gen, device="cuda")
        u = torch.rand((n, 2), generator=gen, device="cuda")
        box = ba[poly]
        state["points"] = (box[:, :2] + u * (box[:, 2:] - box[:, :2])).contiguous()
        state["point_pairs"] = torch.stack([poly, torch.arange(n, device="cuda")], 1).to(torch.int32).contiguous()
    elif kind == "area_plan":
        es, et = a[0][1:] - a[0][:-1], b[0][1:] - b[0][:-1]
        e = (es[pairs[:, 0].long()] + 7) // 8 + (et[pairs[:, 1].long()] + 7) // 8
        state["plan"] = st.area_plan(max_pairs=len(pairs), max_items=int(e.sum()) + 64)
    elif kind == "score":
        par = _grad_inputs({"rows": 1}, seed)[0]
        st.mlp_load(par.cpu().numpy())
    torch.cuda.synchronize()
    return state


def run(state: dict):
    kind, st = state["kind"], state["store"]
    if kind == "query":
        return st.intersect(state["pairs"], mode=state["mode"])
    if kind == "join":
        st.load(0, *state["source"])
        st.load(1, *state["target"])
        st.rasterize(**state["opts"])
        pairs = st.mbr_join(device="cuda") if state["device"] else st.mbr_join()
        state["cand"][:len(pairs)] = pairs
        _, found = st.intersect(pairs, out=state["flags"][:len(pairs)])
        return state["cand"], state["flags"], len(pairs), found
    if kind == "contain":
        return (*st.contain(state["pairs"]), *st.contain_points(state["points"], state["point_pairs"]))
    if kind == "within_join":
        st.load(0, *state["source"])
        st.rasterize(**state["opts"])
        pairs = st.mbr_join(expand=10.0, geography=True, self_join=True)
        state["cand"][:len(pairs)] = pairs
        _, found = st.within(pairs, distance=10.0, geography=True, self_join=True, out=state["flags"][:len(pairs)])
        return state["cand"], state["flags"], len(pairs), found
    if kind == "within_query":
        return st.within(state["pairs"], distance=10.0, geography=False, self_join=True)
    if kind == "area_join":
        st.load(0, *state["source"])
        st.load(1, *state["target"])
        st.rasterize(**state["opts"])
        return st.intersection_area(state["pairs"])
    if kind == "area_plan":
        return state["plan"].run(state["pairs"])
    if kind == "score":
        return st.mlp_predict(state["pairs"])
    return st.mlp_grad(state["x"], state["y"], state["n"])


# ------------------------------------------------------------ what is needed --
def work(case: dict) -> dict:
    """Bytes: each ring, pair or feature read once and each result written once.
    Operations: of a rasterization, 16 per edge for its cells and line, 8 per
    edge for the clip and the area sum; of a pair query, one segment test of 28
    per candidate pair; of an area, 28 per edge of the pair's boundaries; of the
    scorer, its multiply-adds."""
    kind = case["kind"]
    if kind == "grad":
        n = case["rows"]
        par = HID * IN_PAD + HID * HID + 3 * HID + 1
        # forward, and backward's two products (the first layer's inputs need no gradient)
        return {"bytes": 2 * n * IN + n + 8 * par, "flops": 2 * n * (2 * IN * HID + 3 * HID * HID + 3 * HID)}
    nv = _mean_nv(case["n_lo"], case["n_hi"])
    polys = case["n"] if "n" in case else case["ns"] + case["nt"]
    v = polys * nv
    if kind == "join":
        p = 15.0 * case["ns"] * case["nt"] / case["side"] ** 2
        return {"bytes": 8 * v + 9 * p, "flops": 24 * v + 28 * p}
    if kind == "within_join":
        p = 15.0 * case["n"] ** 2 / case["side"] ** 2
        return {"bytes": 8 * v + 9 * p, "flops": 24 * v + 28 * p}
    if kind == "within_query":
        p = case["pairs"]
        return {"bytes": 8 * v + 9 * p, "flops": 28 * p}
    p = case["pairs"]
    if kind == "contain":
        return {"bytes": 8 * min(v, nv * (p + case["points"])) + 9 * p + 17 * case["points"],
                "flops": 28 * p + 8 * case["points"]}
    if kind == "score":
        return {"bytes": 12 * p + 2 * (HID * IN + HID * HID), "flops": 2 * p * (IN * HID + HID * HID + HID)}
    if kind == "area_join":
        return {"bytes": 8 * v + 16 * p, "flops": 24 * v + 56 * nv * p}
    if kind == "area_plan":
        return {"bytes": 8 * v + 16 * p, "flops": 56 * nv * p}
    return {"bytes": 8 * min(v, 2 * nv * p) + 9 * p, "flops": 28 * p}  # query


# --------------------------------------------------------------- in 64 bits --
def _signed_area(r):
    x, y = r[:, 0], r[:, 1]
    return 0.5 * torch.sum(x[:-1] * y[1:] - x[1:] * y[:-1])


def _inside_part(m, o, sign_o):
    """1/2 of the integral of x dy - y dx over ring m's parts inside ring o."""
    total = torch.zeros((), dtype=torch.float64, device=m.device)
    c, g = o[:-1], o[1:] - o[:-1]
    step = max(1, (1 << 24) // len(c))
    for k in range(0, len(m) - 1, step):
        p, q = m[k:k + step + 1][:-1], m[k:k + step + 1][1:]
        d = q - p
        den = d[:, None, 0] * g[None, :, 1] - d[:, None, 1] * g[None, :, 0]
        rx, ry = c[None, :, 0] - p[:, None, 0], c[None, :, 1] - p[:, None, 1]
        safe = torch.where(den == 0, torch.ones_like(den), den)
        t = (rx * g[None, :, 1] - ry * g[None, :, 0]) / safe
        u = (rx * d[:, None, 1] - ry * d[:, None, 0]) / safe
        hit = (den != 0) & (t >= 0) & (t < 1) & (u >= 0) & (u < 1)
        # leaving where the interior of o lies on the other side of its edge
        s = torch.where(sign_o * den > 0, t, -t)
        length = torch.sum(torch.where(hit, s, torch.zeros_like(s)), 1)
        # is the edge's end inside o: parity of o's edges to its right
        y0, y1 = c[None, :, 1], c[None, :, 1] + g[None, :, 1]
        span = (y0 > q[:, None, 1]) != (y1 > q[:, None, 1])
        xi = c[None, :, 0] + (q[:, None, 1] - y0) * g[None, :, 0] / torch.where(span, y1 - y0, torch.ones_like(y0))
        end_in = torch.sum(span & (xi > q[:, None, 0]), 1) % 2
        length = length + end_in
        total = total + torch.sum((p[:, 0] * d[:, 1] - p[:, 1] * d[:, 0]) * length)
    return 0.5 * total


def _exact_areas(case: dict, seed: int):
    gen = _generator(seed)
    a, b = _two_sets(case, gen)
    pairs = _pairs(gen, _boxes(*a), _boxes(*b), case["pairs"]).cpu().numpy()
    oa, ob = a[0].cpu().numpy(), b[0].cpu().numpy()
    out = torch.zeros(len(pairs), dtype=torch.float64, device="cuda")
    for k, (i, j) in enumerate(pairs):
        s, t = a[1][oa[i]:oa[i + 1]].double(), b[1][ob[j]:ob[j + 1]].double()
        s, t = s - s[0].clone(), t - s[0].clone()
        fs, ft = torch.sign(_signed_area(s)), torch.sign(_signed_area(t))
        out[k] = torch.abs(fs * _inside_part(s, t, ft) + ft * _inside_part(t, s, fs))
    return out


def _exact_grad(case: dict, seed: int):
    par, x, y = _grad_inputs(case, seed)
    n = case["rows"]
    par = par.double()
    sizes = [HID * IN_PAD, HID * HID, HID, HID, HID, 1]
    w1, w2, b1, b2, w3, b3 = [t.clone().requires_grad_() for t in torch.split(par, sizes)]
    x, y = x[:n].double(), y[:n].double()

    def gelu(v):
        return 0.5 * v * (1.0 + torch.erf(v / math.sqrt(2.0)))

    h = gelu(x @ w1.view(HID, IN_PAD).T + b1)
    h = gelu(h @ w2.view(HID, HID).T + b2)
    z = h @ w3 + b3
    loss = torch.mean(torch.clamp(z, min=0.0) - z * y + torch.log1p(torch.exp(-torch.abs(z))))
    loss.backward()
    grad = torch.cat([t.grad.flatten() for t in (w1, w2, b1, b2, w3, b3)])
    return float(loss.detach()), grad.cpu().numpy()


def exact(case: dict, seed: int):
    """Areas and gradients; the other kinds return flags, counts and pairs, and
    the scorer's probabilities hang on the rasters of the pairs' polygons."""
    if case["kind"] == "area_join":
        return _exact_areas(case, seed).cpu().numpy()
    if case["kind"] == "area_plan" and case["pairs"] * _mean_nv(8, case["n_hi"]) ** 2 < 2e10:
        return _exact_areas(case, seed)
    if case["kind"] == "grad":
        return _exact_grad(case, seed)
    return None
