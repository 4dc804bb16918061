"""Tile visits by runs and columns at the edges of their ranges: layer counts on
both sides of each instantiation, tiles cut by the lattice on either axis,
every schedule, adjacent and column vias, seeds whose planar edges are all
blocked (only their via column leaves the cell).  Distances bit for bit
against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle as O  # noqa: E402
from orthoroute_b200.lattice import build_lattice, uniform_weights  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

REFERENCE = dict(planar="inner", vias="full", duplicate_vias=True)


def _case(dims, kw, seed):
    lat = build_lattice(*dims, **kw)
    w = uniform_weights(lat, seed=seed, blocked_frac=0.25)
    src = np.random.default_rng(seed).integers(0, lat.N, 5).astype(np.int32)
    s = int(src[0])  # this one can leave its cell by vias only
    row = slice(lat.indptr[s], lat.indptr[s + 1])
    w[row] = np.where(lat.edge_kind[row] == 1, np.float32(3.0), np.float32(np.inf))
    return lat, w, src


# the owner schedule, and the queue schedules with one and two CTAs per SM
@pytest.mark.parametrize("own,spec,per_sm", [("1", "0", "1"), ("0", "0", "1"), ("0", "0", "2"), ("0", "1", "1"),
                                             ("0", "1", "2")])
@pytest.mark.parametrize("dims,kw", [
    ((17, 16, 3), {}), ((33, 47, 6), {}), ((5, 40, 7), {}), ((40, 5, 12), {}), ((31, 33, 13), {}), ((16, 32, 18), {}),
    ((20, 18, 19), {}), ((18, 35, 4), REFERENCE), ((33, 17, 7), REFERENCE), ((21, 20, 16), REFERENCE),
])
def test_distances_at_layer_and_tile_edges(dims, kw, own, spec, per_sm, monkeypatch):
    lat, w, src = _case(dims, kw, seed=sum(dims))
    monkeypatch.setenv("ORSP_LAT_OWN", own)
    monkeypatch.setenv("ORSP_LAT_SPEC", spec)
    monkeypatch.setenv("ORSP_LAT_BLOCKS_PER_SM", per_sm)
    dg = DeviceGraph.from_lattice(lat)
    wt = torch.from_numpy(w).cuda()
    many = torch.empty(len(src), lat.N, device="cuda")
    dg.sssp_sources(wt, src, many)
    one = torch.empty(lat.N, device="cuda")
    for k, s in enumerate(src.tolist()):
        _, ref, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [s])
        dg.sssp(wt, s, -1, dist_out=one)
        assert np.array_equal(one.cpu().numpy().view(np.uint32), ref.view(np.uint32))
        assert np.array_equal(many[k].cpu().numpy().view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("dims,kw", [
    ((592, 64, 3), {}),       # 148 tiles: one per SM
    ((593, 64, 3), {}),       # 152: two CTAs per SM from here
    ((196, 210, 18), {}), ((230, 250, 9), {}), ((200, 180, 5), REFERENCE),
    ((592, 128, 3), {}),      # 296: the last owned launch
    ((593, 128, 3), {}),      # 304: queue
])
def test_distances_at_owner_schedule_limits(dims, kw):
    lat, w, src = _case(dims, kw, seed=sum(dims))
    dg = DeviceGraph.from_lattice(lat)
    wt = torch.from_numpy(w).cuda()
    one = torch.empty(lat.N, device="cuda")
    for s in src[:3].tolist():
        _, ref, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [s])
        dg.sssp(wt, s, -1, dist_out=one)
        assert np.array_equal(one.cpu().numpy().view(np.uint32), ref.view(np.uint32))
