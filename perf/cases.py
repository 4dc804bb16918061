"""Measured workloads of the PathFinder hot path.

Each case is a call that a routing program makes, through the entry points it
would use, on inputs drawn from the case's seed: net searches, the drop-in
calls of the reference router, whole-graph searches, batched searches, the
negotiation loop, the per-iteration accounting, and the layers of the
learned warm start.

A routing program builds its lattice and the graph handle once and keeps
them; `prepare` does the same, through a small table of the last few lattices.
Everything that a routing call changes from net to net - costs, nets, boxes,
histories, activations - is made again for each seed.
"""
from __future__ import annotations

import math
from collections import OrderedDict

import numpy as np
import torch

from orthoroute_b200 import _lib
from orthoroute_b200.accounting import DeviceEdgeAccountant
from orthoroute_b200.dropin import DropInSet
from orthoroute_b200.lattice import bbox_with_margin, board_footprints, build_lattice, layer_directions, random_boxes
from orthoroute_b200.negotiate import NegotiationConfig, PathFinder
from orthoroute_b200.solver import DeviceGraph

KEPT = 4  # lattices kept at a time
_kept: OrderedDict = OrderedDict()


def listed():
    return [
        # one net after another on a small board (the 100 x 100 x 4 plain
        # board): the search of a short net, where latency is all there is
        {"name": "net_small", "kind": "net", "nx": 100, "ny": 100, "nz": 4, "nets": 4, "span": 40, "margin": 10},
        # the same on the 600 x 600 x 18 backplane: boxes of the nets that
        # join two connectors
        {"name": "net_backplane", "kind": "net", "nx": 600, "ny": 600, "nz": 18, "nets": 4, "span": 500, "margin": 10},
        # the reference router's own calls per net (ROI, search, path to
        # edges) on the graph that its Lattice3D builds: any-layer vias, each twice
        {"name": "dropin_lattice3d", "kind": "dropin", "graph": "lattice3d", "nx": 200, "ny": 200, "nz": 6, "nets": 4,
         "portals": False},
        # one source, distances to every node
        {"name": "full_search", "kind": "sources", "nx": 600, "ny": 600, "nz": 12, "sources": 1},
        # many sources on one cost array (the 1000 x 1000 x 12 scaling lattice)
        {"name": "sources_many", "kind": "sources", "nx": 1000, "ny": 1000, "nz": 12, "sources": 16},
        # searches of uneven boxes in one call, with the default plan and with
        # the tile sweeps that the autotuner settles on (the batch sweep's boxes)
        {"name": "batch_default", "kind": "batch", "nx": 400, "ny": 400, "nz": 16, "searches": 512, "plan": "default"},
        {"name": "batch_sweeps", "kind": "batch", "nx": 400, "ny": 400, "nz": 16, "searches": 2048, "plan": "sweeps"},
        # the negotiation loop, one net at a time, on the plain board
        {"name": "route_plain", "kind": "route", "nx": 100, "ny": 100, "nz": 4, "nets": 200, "iterations": 2,
         "groups": 0, "mode": "sequential"},
        # the first iteration of a backplane board in snapshot groups
        {"name": "route_groups", "kind": "route", "nx": 600, "ny": 600, "nz": 18, "nets": 1000, "iterations": 1,
         "groups": 32, "mode": "batched"},
        # what one negotiation iteration does to the backplane's edge arrays
        {"name": "accounting", "kind": "accounting", "edges": 25_178_400, "bias": True},
        # a 32 to 32 channel layer of the warm-start network on a board, and
        # its gradients on a training window
        {"name": "warm_conv", "kind": "conv", "d": 18, "h": 400, "w": 400, "cin": 32, "cout": 32, "relu": True,
         "grad": False},
        {"name": "warm_grad", "kind": "conv", "d": 18, "h": 200, "w": 200, "cin": 32, "cout": 32, "relu": True,
         "grad": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["net", "net", "dropin", "sources", "batch", "batch", "route", "route", "accounting", "conv"])
    if kind == "net":
        nx, ny, nz = _log(rng, 60, 600), _log(rng, 60, 600), rng.randint(2, 18)
        nz = 3 if nz == 2 else nz
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "nets": rng.randint(1, 6),
                "span": _log(rng, 8, max(9, min(nx, ny) - 1)), "margin": rng.choice([4, 10, 20])}
    if kind == "dropin":
        return {"kind": kind, "graph": rng.choice(["lattice3d", "adjacent"]), "nx": _log(rng, 60, 300),
                "ny": _log(rng, 60, 300), "nz": rng.randint(4, 8), "nets": rng.randint(1, 4),
                "portals": rng.random() < 0.4}
    if kind == "sources":
        n = _log(rng, 1, 16)
        side = 700 if n > 4 else 900
        return {"kind": kind, "nx": _log(rng, 100, side), "ny": _log(rng, 100, side), "nz": rng.randint(3, 12),
                "sources": n}
    if kind == "batch":
        plan = rng.choice(["default", "sweeps"])
        return {"kind": kind, "nx": rng.randint(150, 400), "ny": rng.randint(150, 400), "nz": rng.randint(6, 16),
                "searches": _log(rng, 16, 512 if plan == "default" else 2048), "plan": plan}
    if kind == "route":
        groups = rng.choice([0, 8, 32])
        nx, ny = _log(rng, 80, 240), _log(rng, 80, 240)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": rng.randint(4, 12),
                "nets": max(16, min(200, nx * ny // 60)), "iterations": rng.randint(1, 2), "groups": groups,
                "mode": "batched" if groups else rng.choice(["sequential", "batched"])}
    if kind == "accounting":
        return {"kind": kind, "edges": _log(rng, 50_000, 25_000_000), "bias": rng.random() < 0.5}
    grad = rng.random() < 0.5
    side = 200 if grad else 400
    cin, cout = rng.choice([(16, 32), (32, 32), (32, 16)])
    return {"kind": "conv", "d": rng.randint(4, 18), "h": 8 * rng.randint(3, side // 8), "w": 8 * rng.randint(3, side // 8),
            "cin": cin, "cout": cout, "relu": rng.random() < 0.8, "grad": grad}


# ------------------------------------------------------------------ inputs
def _keep(key, make):
    """The object of `key`, built on first use; the oldest goes when KEPT are held."""
    if key in _kept:
        _kept.move_to_end(key)
    else:
        while len(_kept) >= KEPT:
            _kept.popitem(last=False)
        _kept[key] = make()
    return _kept[key]


def _lattice(nx, ny, nz, graph="adjacent"):
    if graph == "lattice3d":
        return build_lattice(nx, ny, nz, planar="inner", vias="full", duplicate_vias=True)
    return build_lattice(nx, ny, nz)


def _graph(case):
    """(lattice, device graph, via mask on the device) of a case's board."""
    nx, ny, nz, graph = case["nx"], case["ny"], case["nz"], case.get("graph", "adjacent")

    def make():
        lat = _lattice(nx, ny, nz, graph)
        via = torch.from_numpy(lat.edge_kind).cuda() == 1
        if case["kind"] == "dropin":
            return lat, DropInSet(lat.indptr, lat.indices, lattice=lat, nx=nx, ny=ny, nz=nz), via
        return lat, DeviceGraph.from_lattice(lat), via

    return _keep((case["kind"] == "dropin", nx, ny, nz, graph), make)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _uniform_costs(via, seed, blocked):
    """Planar edges uniform in [1, 2), vias 3, a share of all edges blocked."""
    g = _generator(seed)
    w = 1.0 + torch.rand(via.numel(), generator=g, device="cuda")
    w[via] = 3.0
    w[torch.rand(via.numel(), generator=g, device="cuda") < blocked] = math.inf
    return w


def _negotiated_costs(lat, seed):
    """The costs that the searches of a running negotiation see: the base
    costs, present congestion on a few edges, a history on others, and the
    router's index jitter."""
    g = _generator(seed)
    w = torch.from_numpy(lat.base_cost).cuda()
    r = torch.rand(lat.E, generator=g, device="cuda")
    w = w + torch.where(r < 0.06, 1.125, 0.0)
    h = torch.rand(lat.E, generator=g, device="cuda")
    w = w + torch.where(h < 0.04, 1.0 + torch.floor(h * 100.0), torch.zeros_like(h))
    i = torch.arange(lat.E, device="cuda").remainder(9973).float()
    return (w + i * 1e-6).float().contiguous()


def _nets(rng, case, count):
    """Two-pin nets on the top layer, at most `span` cells apart in x and y."""
    nx, ny, span = case["nx"], case["ny"], case.get("span", 10**9)
    x = rng.integers(0, nx, count)
    y = rng.integers(0, ny, count)
    u = np.clip(x + rng.integers(-span, span + 1, count), 0, nx - 1)
    v = np.clip(y + rng.integers(-span, span + 1, count), 0, ny - 1)
    u = np.where((u == x) & (v == y), (u + 1) % nx, u)
    return (y * nx + x).astype(np.int32), (v * nx + u).astype(np.int32)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"case": case}
    if kind == "net":
        lat, s["graph"], _ = _graph(case)
        s["cost"] = _negotiated_costs(lat, seed)
        s["src"], s["dst"] = _nets(rng, case, case["nets"])
        s["box"] = bbox_with_margin(lat, s["src"], s["dst"], case["margin"])
    elif kind == "dropin":
        lat, s["set"], _ = _graph(case)
        s["cost"] = _negotiated_costs(lat, seed)
        s["src"], s["dst"] = _nets(rng, case, case["nets"])
        s["nx"], s["plane"] = case["nx"], case["nx"] * case["ny"]
    elif kind == "sources":
        lat, s["graph"], via = _graph(case)
        s["cost"] = _uniform_costs(via, seed, 0.05)
        s["sources"] = rng.integers(0, lat.N, case["sources"]).astype(np.int32)
        s["dist"] = torch.empty(case["sources"], lat.N, dtype=torch.float32, device="cuda")
    elif kind == "batch":
        lat, s["graph"], via = _graph(case)
        s["cost"] = _uniform_costs(via, seed, 0.03)
        box, src, dst = random_boxes(lat, case["searches"], seed=seed, lo=(20, 20, 4), hi=(case["nx"], case["ny"], case["nz"]))
        s["src"], s["dst"], s["box"] = (torch.from_numpy(a).cuda() for a in (src, dst, box))
        s["plan"] = [{"max_nodes": 1 << 40, "impl": 1, "tile_w": 32}] if case["plan"] == "sweeps" else None
    elif kind == "route":
        cfg = NegotiationConfig(max_iterations=case["iterations"], cost_update="net", reroute="offenders",
                                roi_margin=10, full_graph_retry=False, net_order="disjoint", stall_grow=10,
                                group_nets=case["groups"], group_repair=3 if case["groups"] else 0)
        s["router"] = _keep(("route", case["nx"], case["ny"], case["nz"], case["groups"], case["iterations"]),
                            lambda: PathFinder(_lattice(case["nx"], case["ny"], case["nz"]), config=cfg))
        if case["nx"] >= 300:  # pins of connector footprints, as on a backplane
            s["src"], s["dst"] = _footprint_nets(case, seed)
        else:
            cells = rng.choice(case["nx"] * case["ny"], size=2 * case["nets"], replace=False).astype(np.int32)
            s["src"], s["dst"] = cells[:case["nets"]].copy(), cells[case["nets"]:].copy()
    elif kind == "accounting":
        E, g = case["edges"], _generator(seed)
        acc = DeviceEdgeAccountant(E)
        r = torch.rand(E, generator=g, device="cuda")
        acc.usage.copy_(torch.where(r < 0.1, (r * 40).int() + 1, 0))
        h = torch.rand(E, generator=g, device="cuda")
        acc.history.copy_(torch.where(h < 0.05, h * 60, 0.0))
        acc.present_ema.copy_(torch.where(r < 0.1, r * 30, 0.0))
        s["acc"] = acc
        via = torch.rand(E, generator=g, device="cuda") < 0.47
        s["base"] = torch.where(via, 3.0, 1.0).float()
        if case["bias"]:
            s["kind"] = via.to(torch.uint8)
            s["layer"] = torch.randint(0, 18, (E,), generator=g, device="cuda", dtype=torch.uint8)
            s["bias"] = (0.8 + 0.5 * torch.rand(18, generator=g, device="cuda")).float()
    else:
        g = _generator(seed)
        d, h, w, cin, cout = (case[k] for k in ("d", "h", "w", "cin", "cout"))
        s["x"] = torch.relu(torch.randn(d, h, w, cin, generator=g, device="cuda")).to(torch.bfloat16)
        s["wf"] = torch.randn(27, cin, cout, generator=g, device="cuda") * math.sqrt(2.0 / (27 * cin))
        s["b"] = torch.randn(cout, generator=g, device="cuda") * 0.1
        # the layer's weights as its kernels read them, laid out once
        s["wt"] = torch.empty(27 * cin * cout, dtype=torch.bfloat16, device="cuda")
        _call("orsp_warm_pack_weights", s["wf"], s["wt"], cin, cout, 0)
        if case["grad"]:
            s["wt_t"] = torch.empty(27 * cin * cout, dtype=torch.bfloat16, device="cuda")
            _call("orsp_warm_pack_weights", s["wf"], s["wt_t"], cin, cout, 1)
            s["y"] = torch.relu(torch.randn(d, h, w, cout, generator=g, device="cuda")).to(torch.bfloat16)
            s["dy"] = torch.randn(d, h, w, cout, generator=g, device="cuda").to(torch.bfloat16)
    return s


def _footprint_nets(case, seed):
    """The nets of board_footprints on a lattice shell (the pins need only its sides)."""
    b = board_footprints(case["nx"], case["ny"], 1, case["nets"], None, seed=seed)
    return b.src, b.dst


# ------------------------------------------------------------------ passes
def _call(name, *args):
    """A kernel of the warm-start network through the C ABI."""
    a = [_lib.ptr(v) if isinstance(v, torch.Tensor) or v is None else v for v in args]
    _lib.check(getattr(_lib.load(), name)(*a, int(torch.cuda.current_stream().cuda_stream)), name)


def _rows(case, paths):
    """Lists of node or edge ids as the rows of one array, -1 past their ends, with their lengths."""
    lens = np.asarray([0 if p is None else len(p) for p in paths], np.int32)
    rows = np.full((len(paths), 2 * (case["nx"] + case["ny"]) + 16 * case["nz"]), -1, np.int32)
    for k, p in enumerate(paths):
        rows[k, :lens[k]] = p if lens[k] else -1
    return {"rows": rows, "lens": lens}


def _trace(case, r):
    """The (sum, count) of overused edges per iteration, zeros after the last one made."""
    t = [tuple(v) for v in r.overuse_trace()]
    return t + [(0, 0)] * (case["iterations"] - len(t))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "net":
        out = []
        for k in range(case["nets"]):
            _, path, _ = s["graph"].sssp_box(s["cost"], int(s["src"][k]), int(s["dst"][k]), s["box"][k], path_cap=8192)
            out.append(None if path is None else path.cpu().numpy())
        return _rows(case, out)
    if kind == "dropin":
        d, paths, edges, sizes = s["set"], [], [], []
        for a, b in zip(s["src"].tolist(), s["dst"].tolist()):
            seeds = None
            if case["portals"]:  # each pin may be left on any inner layer, at the cost of the barrel
                seeds = [(z * s["plane"] + n, 3.0 + 0.45 * (z - 1)) for n in (a, b) for z in range(1, case["nz"] - 1)]
            roi, g2r = d.extract_roi(a, b, portal_seeds=seeds)
            if seeds:
                half = len(seeds) // 2
                got = d.solver.find_path_multisource_multisink(seeds[:half], seeds[half:], s["cost"], roi, g2r)
                path = got[0] if got else None
            else:
                path = d.find_path_roi(a, b, s["cost"], roi, g2r)
            paths.append(path)
            edges.append(d.path_to_edges(path) if path else None)
            sizes.append(len(roi))
        return {"path": _rows(case, paths), "edges": _rows(case, edges), "roi": np.asarray(sizes, np.int64)}
    if kind == "sources":
        if case["sources"] == 1:
            s["graph"].sssp(s["cost"], int(s["sources"][0]), -1, dist_out=s["dist"][0])
        else:
            s["graph"].sssp_sources(s["cost"], s["sources"], s["dist"])
        return s["dist"]
    if kind == "batch":
        s["graph"].set_batch_plan(s["plan"])
        nodes, edges, lens = s["graph"].batch_bbox(s["cost"], s["src"], s["dst"], s["box"], path_cap=2048)
        # rows are defined up to their lengths
        at = torch.arange(nodes.shape[1], device="cuda")[None, :]
        return {"nodes": nodes.masked_fill_(at >= lens[:, None], -1),
                "edges": edges.masked_fill_(at >= lens[:, None] - 1, -1), "lens": lens}
    if kind == "route":
        r = s["router"].route(s["src"], s["dst"], mode=case["mode"])
        return {"paths": _rows(case, r.paths), "usage": r.edge_usage, "wirelength": r.wirelength, "vias": r.vias,
                "overuse": np.asarray(_trace(case, r), np.int64)}
    if kind == "accounting":
        acc, more = s["acc"], {}
        if case["bias"]:
            more = {"edge_layer": s["layer"], "layer_bias_per_layer": s["bias"], "edge_kind": s["kind"]}
        acc.refresh_from_canonical()
        acc.update_present_ema(beta=0.4)
        acc.update_costs(s["base"], 1.125, 1.0, add_jitter=True, base_cost_weight=1.0, **more)
        total, count = acc.compute_overuse()
        acc.update_history(1.0, base_costs=s["base"], history_cap_multiplier=15.0, decay_factor=0.98, use_raw_present=True)
        return {"cost": acc.total_cost, "ema": acc.present_ema, "history": acc.history, "overuse": total, "count": count}
    d, h, w, cin, cout = (case[k] for k in ("d", "h", "w", "cin", "cout"))
    if not case["grad"]:
        y = torch.empty(d, h, w, cout, dtype=torch.bfloat16, device="cuda")
        _call("orsp_warm_conv3d_tc", s["x"], None, s["wt"], s["b"], y, None, d, h, w, cin, cout, int(case["relu"]))
        return y
    mask = s["y"] if case["relu"] else None
    dw = torch.zeros(27, cin, cout, device="cuda")
    db = torch.zeros(cout, device="cuda")
    _call("orsp_warm_wgrad_tc", s["x"], s["dy"], mask, dw, db, d, h, w, cin, cout)
    dx = torch.empty(d, h, w, cin, dtype=torch.bfloat16, device="cuda")
    _call("orsp_warm_conv3d_tc", s["dy"], mask, s["wt_t"], None, dx, None, d, h, w, cout, cin, 0)
    return {"dw": dw, "db": db, "dx": dx}


# ------------------------------------------------------------------ what a pass cannot do without
def _adjacent_edges(nx, ny, nz):
    h = sum("h" in a for a in layer_directions(nz))
    v = sum("v" in a for a in layer_directions(nz))
    return 2 * (h * (nx - 1) * ny + v * nx * (ny - 1) + nx * ny * (nz - 1))


def work(case):
    kind = case["kind"]
    if kind == "net":
        # the mean box of its nets: every edge's cost once, one add per edge
        side = min(case["span"] / 2, min(case["nx"], case["ny"]) / 3) + 2 * case["margin"]
        w, h = min(side, case["nx"]), min(side, case["ny"])
        e = case["nets"] * _adjacent_edges(int(w), int(h), case["nz"])
        return {"bytes": 4 * e, "flops": e}
    if kind == "dropin":
        e = case["nets"] * min(50_000, case["nx"] * case["ny"] * case["nz"]) * 6
        return {"bytes": 8 * e, "flops": e}
    if kind == "sources":
        n, e = case["nx"] * case["ny"] * case["nz"], _adjacent_edges(case["nx"], case["ny"], case["nz"])
        return {"bytes": 4 * e + 4 * n * case["sources"], "flops": e * case["sources"]}
    if kind == "batch":
        # the costs of the lattice once; half of each box lies nearer than its target
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        mean = [(b - a) / math.log(b / a) if b > a else a for a, b in ((20, nx), (20, ny), (4, nz))]
        e = case["searches"] * _adjacent_edges(*(int(v) for v in mean)) // 2
        return {"bytes": 4 * _adjacent_edges(nx, ny, nz), "flops": e}
    if kind == "route":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        # the edge arrays (base, capacity, history, usage, cost) once an iteration, each net's box once
        e = case["nets"] * _adjacent_edges(min(nx, nx // 3 + 20), min(ny, ny // 3 + 20), nz) * case["iterations"]
        return {"bytes": 20 * _adjacent_edges(nx, ny, nz) * case["iterations"], "flops": e}
    if kind == "accounting":
        # usage, base, capacity read; present, ema, history read and written; costs written
        return {"bytes": (10 * 4 + (2 if case["bias"] else 0)) * case["edges"], "flops": 20 * case["edges"]}
    vox = case["d"] * case["h"] * case["w"]
    mul = 2 * 27 * case["cin"] * case["cout"] * vox
    if case["grad"]:  # input, both output-side maps read; input gradient written
        return {"bytes": 2 * vox * (2 * case["cin"] + (2 if case["relu"] else 1) * case["cout"]), "flops": 2 * mul}
    return {"bytes": 2 * vox * (case["cin"] + case["cout"]), "flops": mul}


# ------------------------------------------------------------------ in 64 bits
def _exact_distances(case, seed):
    """Distances from each source by repeated relaxation of every edge in float64."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    lat, _, via = _graph(case)
    cost = _uniform_costs(via, seed, 0.05).double()
    src = np.random.default_rng(seed).integers(0, lat.N, case["sources"]).astype(np.int32)
    node = torch.repeat_interleave(torch.arange(lat.N, device="cuda"),
                                   torch.from_numpy(np.diff(lat.indptr).astype(np.int64)).cuda())
    step = torch.from_numpy(lat.indices).cuda().long() - node
    into = {}
    for d in (1, -1, nx, -nx, nx * ny, -nx * ny):  # weight of the edge that enters v from v - d
        m = step == d
        w = torch.full((lat.N,), math.inf, dtype=torch.float64, device="cuda")
        w[node[m] + d] = cost[m]
        into[d] = w
    del node, step
    dist = torch.full((case["sources"], lat.N), math.inf, dtype=torch.float64, device="cuda")
    dist[torch.arange(case["sources"]), torch.from_numpy(src).long()] = 0.0
    while True:
        before = dist.clone()
        for _ in range(64):
            for d, w in into.items():
                if d > 0:
                    torch.minimum(dist[:, d:], dist[:, :-d] + w[d:], out=dist[:, d:])
                else:
                    torch.minimum(dist[:, :d], dist[:, -d:] + w[:d], out=dist[:, :d])
        if torch.equal(before, dist):
            return dist if case["sources"] > 1 else dist.reshape(1, -1)


def _taps():
    return [(z, y, x) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]


def _shifted(a, tap):
    """a[v + tap], zero outside the grid."""
    z, y, x = tap
    d, h, w = a.shape[:3]
    out = torch.zeros_like(a)
    out[max(0, -z):d - max(0, z), max(0, -y):h - max(0, y), max(0, -x):w - max(0, x)] = \
        a[max(0, z):d - max(0, -z), max(0, y):h - max(0, -y), max(0, x):w - max(0, -x)]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "sources":
        if case["nx"] * case["ny"] * case["nz"] * case["sources"] > 30_000_000:
            return None
        return _exact_distances(case, seed)
    if kind == "accounting":
        s = prepare(case, seed)
        acc = s["acc"]
        present = acc.usage.double()
        beta = float(np.float32(0.4))
        ema = beta * present + float(np.float32(0.6)) * acc.present_ema.double()
        over = (ema - 1.0).clamp(min=0.0)
        jitter = torch.arange(case["edges"], device="cuda").float().double().remainder(9973) * float(np.float32(1e-6))
        bias = torch.ones_like(ema)
        if case["bias"]:
            bias = torch.where(s["kind"] == 0, s["bias"].double()[s["layer"].long()], 1.0)
        cost = s["base"].double() * bias + 1.125 / bias.clamp(min=0.5) * over + acc.history.double() + jitter
        raw = (present - 1.0).clamp(min=0.0)
        history = acc.history.double() * float(np.float32(0.98)) + torch.minimum(raw, 15.0 * s["base"].double())
        return {"cost": cost, "ema": ema, "history": history, "overuse": None, "count": None}
    if kind != "conv":
        return None  # paths, edges and counts: whole numbers
    s = prepare(case, seed)
    d, h, w, cin, cout = (case[k] for k in ("d", "h", "w", "cin", "cout"))
    weights = s["wt"].double().reshape(27, cin, cout)
    x = s["x"].double()
    if not case["grad"]:
        y = s["b"].double().expand(d, h, w, cout).clone()
        for t, tap in enumerate(_taps()):
            y += _shifted(x, tap) @ weights[t]
        return torch.relu(y) if case["relu"] else y
    g = s["dy"].double()
    if case["relu"]:
        g = torch.where(s["y"] > 0, g, 0.0)
    dw = torch.empty(27, cin, cout, dtype=torch.float64, device="cuda")
    dx = torch.zeros(d, h, w, cin, dtype=torch.float64, device="cuda")
    flat = g.reshape(-1, cout)
    for t, tap in enumerate(_taps()):
        dw[t] = _shifted(x, tap).reshape(-1, cin).T @ flat
        dx += _shifted(g, tuple(-k for k in tap)) @ weights[t].T
    return {"dw": dw, "db": flat.sum(0), "dx": dx}
