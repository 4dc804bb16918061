"""The backtrace at the edges of its rounds: straight runs and via stacks around
the number of cells a round covers, many equal paths, zero-cost edges towards
higher ids (the rank decides), adjacent and column vias.  Paths and lengths equal the
oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle as O  # noqa: E402
from orthoroute_b200.lattice import build_lattice  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

REFERENCE = dict(planar="inner", vias="full", duplicate_vias=True)


def _path(dg, wt, s, t):
    path = dg.sssp(wt, s, t)[1]
    return [] if path is None else path.cpu().tolist()


@pytest.mark.parametrize("dims,kw", [((75, 20, 2), {}), ((20, 75, 6), {}), ((24, 24, 12), {}), ((1, 9, 7), {}),
                                     ((40, 30, 5), REFERENCE), ((22, 26, 18), REFERENCE)])
@pytest.mark.parametrize("low", [0, 1])
def test_paths_with_ties_and_long_runs(dims, kw, low):
    lat = build_lattice(*dims, **kw)
    rng = np.random.default_rng(sum(dims) + low)
    dg = DeviceGraph.from_lattice(lat)
    via = lat.edge_kind == 1
    up = np.repeat(np.arange(lat.N), np.diff(lat.indptr)) < lat.indices
    for kind in ("flat", "few", "cheap vias"):
        w = np.ones(lat.E, np.float32)  # flat: ties everywhere
        if kind != "flat":
            w = rng.integers(1, 4, lat.E).astype(np.float32)
            if kind == "cheap vias":
                w[via] = 0.25
            if low == 0:
                w[up & (rng.random(lat.E) < 0.5)] = 0.0
        wt = torch.from_numpy(w).cuda()
        for _ in range(6):
            s, t = (int(v) for v in rng.integers(0, lat.N, 2))
            path, _, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [s], dst=t)
            assert _path(dg, wt, s, t) == path.tolist()


@pytest.mark.parametrize("run", [1, 2, 13, 14, 15, 16, 30, 31, 32, 33, 45, 46])
def test_run_lengths(run):
    # cheap edges along x on layer 0 (or 2), then up the stack and along y
    lat = build_lattice(64, 64, 6)
    src = np.repeat(np.arange(lat.N), np.diff(lat.indptr))
    x, y = src % 64, src // 64 % 64
    w = np.full(lat.E, 50.0, np.float32)
    w[lat.edge_kind == 1] = 1.0
    w[(y == 3) & (x <= 3 + run)] = 1.0
    w[(x == 3 + run) & (y >= 3)] = 1.0
    dg = DeviceGraph.from_lattice(lat)
    wt = torch.from_numpy(w).cuda()
    s = 3 * 64 + 3
    for zt in (0, 1, 3, 5):
        t = (zt * 64 + 3 + run) * 64 + 3 + run
        path, _, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [s], dst=t)
        assert _path(dg, wt, s, t) == path.tolist()
        back, _, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [t], dst=s)
        assert _path(dg, wt, t, s) == back.tolist()
