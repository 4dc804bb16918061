"""Box searches whose walk uses the parents recorded by the search against the
same searches with distances asked for, whose walk reads them: one tile, tiles
cut by the box, odd and single layers, the largest boxes whose parents are
recorded and the first beyond, ties, zero costs, blocked and NaN edges, targets
cut off, equal ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200._lib import OrspError  # noqa: E402
from orthoroute_b200.lattice import build_lattice  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402


def _search(dg, w, src, dst, box, dist_out):
    """(status, path); a plateau of zero costs may have no parent of smaller id, which is an error."""
    try:
        status, path, _ = dg.sssp_box(w, src, dst, box, dist_out=dist_out, path_cap=8192)
    except OrspError as e:
        return e.status, np.zeros(0, np.int32)
    return status, np.zeros(0, np.int32) if path is None else path.cpu().numpy().copy()


@pytest.mark.parametrize("dims", [(16, 16, 2), (17, 33, 3), (1, 50, 4), (60, 47, 5), (140, 130, 6), (64, 64, 12),
                                  (150, 160, 18), (160, 170, 18), (250, 240, 5), (40, 40, 1)])
@pytest.mark.parametrize("costs", ["fractional", "ties", "zeros"])
def test_recorded_parents_give_the_walk_on_distances(dims, costs):
    lat = build_lattice(*dims)
    rng = np.random.default_rng(sum(dims))
    w = {"fractional": 1.0 + rng.random(lat.E), "ties": np.where(lat.edge_kind == 1, 3.0, 1.0),
         "zeros": rng.integers(0, 3, lat.E)}[costs].astype(np.float32)
    w[rng.random(lat.E) < 0.04] = np.inf
    w[rng.random(lat.E) < 0.01] = np.nan
    wt = torch.from_numpy(w).cuda()
    dg = DeviceGraph.from_lattice(lat)
    dist = torch.empty(lat.N, dtype=torch.float32, device="cuda")
    hi = np.array(dims) - 1
    for k in range(12):
        a, b = rng.integers(0, hi + 1), rng.integers(0, hi + 1)
        lo3, hi3 = np.maximum(np.minimum(a, b) - 2, 0), np.minimum(np.maximum(a, b) + 2, hi)
        box = np.stack([lo3, hi3], 1).reshape(-1) if k % 3 else np.stack([np.zeros(3, int), hi], 1).reshape(-1)
        if k == 1:
            b = a
        s, d = (int((p[2] * dims[1] + p[1]) * dims[0] + p[0]) for p in (a, b))
        (st1, p1), (st2, p2) = (_search(dg, wt, s, d, box, out) for out in (None, dist))
        assert st1 == st2
        assert np.array_equal(p1, p2)
