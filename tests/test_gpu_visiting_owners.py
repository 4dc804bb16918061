"""The schedule of visiting owners where tiles outnumber the CTAs: a handful of
CTAs (every idle tile is given back), one CTA, and as many as the GPU holds;
layer counts on both sides of each instantiation, cut tiles, adjacent and
column vias, own and shared distances.  Distances bit for bit against the
oracle, batched paths against the one-CTA search."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle as O  # noqa: E402
from orthoroute_b200.lattice import build_lattice, uniform_weights  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

REFERENCE = dict(planar="inner", vias="full", duplicate_vias=True)


def _check(lat, seed, nsrc):
    w = uniform_weights(lat, seed=seed, blocked_frac=0.2)
    src = np.random.default_rng(seed).integers(0, lat.N, nsrc).astype(np.int32)
    dg = DeviceGraph.from_lattice(lat)
    wt = torch.from_numpy(w).cuda()
    many = torch.empty(nsrc, lat.N, device="cuda")
    dg.sssp_sources(wt, src, many)
    one = torch.empty(lat.N, device="cuda")
    for k, s in enumerate(src.tolist()):
        _, ref, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [s])
        dg.sssp(wt, s, -1, dist_out=one)
        assert np.array_equal(one.cpu().numpy().view(np.uint32), ref.view(np.uint32))
        assert np.array_equal(many[k].cpu().numpy().view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("ctas", ["1", "3", "20", "0"])
@pytest.mark.parametrize("dims,kw", [
    ((65, 49, 2), {}), ((33, 130, 6), {}), ((90, 17, 7), {}), ((40, 70, 12), {}), ((70, 40, 13), {}), ((48, 48, 18), {}),
    ((50, 35, 4), REFERENCE), ((33, 50, 8), REFERENCE), ((40, 33, 17), REFERENCE),
])
def test_few_ctas(dims, kw, ctas, monkeypatch):
    monkeypatch.setenv("ORSP_LAT_OWN", "0")
    monkeypatch.setenv("ORSP_LIVE_CTAS", ctas)
    _check(build_lattice(*dims, **kw), sum(dims), 3)


@pytest.mark.parametrize("dims,kw", [((593, 128, 3), {}), ((330, 300, 4), {}), ((320, 310, 5), REFERENCE)])
def test_more_tiles_than_ctas(dims, kw):
    _check(build_lattice(*dims, **kw), sum(dims), 3)


@pytest.mark.parametrize("nbox,side", [(1, 300), (5, 150), (14, 160), (16, 160)])
def test_boxes_around_the_front_limit(nbox, side):
    lat = build_lattice(400, 380, 6)
    w = torch.from_numpy(uniform_weights(lat, seed=nbox, blocked_frac=0.1)).cuda()
    rng = np.random.default_rng(nbox)
    x, y = rng.integers(0, 400 - side, nbox), rng.integers(0, 380 - side, nbox)
    box = np.stack([x, x + side - 1, y, y + side - 1, 0 * x, 0 * x + 5], 1).astype(np.int32)
    src = (y + rng.integers(0, side, nbox)) * 400 + x + rng.integers(0, side, nbox)
    dst = (y + rng.integers(0, side, nbox)) * 400 + x + rng.integers(0, side, nbox)
    dg = DeviceGraph.from_lattice(lat)
    args = [torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda() for a in (src, dst, box)]
    nodes, edges, lens = dg.batch_bbox(w, *args)
    dg.set_batch_plan([{"max_nodes": 1 << 40, "impl": 0}])
    n0, e0, l0 = dg.batch_bbox(w, *args)
    assert torch.equal(lens, l0) and int(lens.max()) > 2
    for k, n in enumerate(lens.tolist()):
        assert torch.equal(nodes[k, :n], n0[k, :n])
        assert torch.equal(edges[k, : max(n - 1, 0)], e0[k, : max(n - 1, 0)])
