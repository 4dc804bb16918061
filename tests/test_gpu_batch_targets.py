"""Batched box searches whose sweeps stop passing on what cannot reach the
target in time, against one CTA per search: equal costs (every path ties, so
the bound is met with equality), integer costs with and without zeros, costs
whose ratio to the path's length is beyond the bound's range, walls that send
the path a long way round, targets cut off, whole-lattice boxes (one gather for
all) and small ones (a gather per box)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200.lattice import build_lattice, random_boxes  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402


def _costs(lat, kind, rng):
    if kind == "equal":
        return np.ones(lat.E, np.float32)
    if kind == "integer":
        return rng.integers(1, 4, lat.E).astype(np.float32)
    if kind == "zeros":
        return rng.integers(0, 2, lat.E).astype(np.float32)
    if kind == "ratio":
        return (10.0 ** rng.uniform(-7, 3, lat.E)).astype(np.float32)
    w = 1.0 + rng.random(lat.E, dtype=np.float32)
    u = np.repeat(np.arange(lat.N), np.diff(lat.indptr))
    x, v = lat.indices % lat.nx, lat.indices
    # walls every six columns, open at one row of alternating ends
    y = v % (lat.nx * lat.ny) // lat.nx
    wall = (x % 6 == 3) & (u != v) & (y != np.where(x // 6 % 2 == 0, 0, lat.ny - 1))
    w[wall] = np.inf
    return w


@pytest.mark.parametrize("kind", ["equal", "integer", "zeros", "ratio", "walls"])
@pytest.mark.parametrize("dims,lo", [((120, 110, 3), (60, 60, 3)), ((70, 65, 9), (16, 16, 2)), ((90, 90, 18), (90, 90, 18)),
                                     ((40, 200, 1), (17, 33, 1))])
def test_sweeps_with_targets_equal_one_cta_per_search(kind, dims, lo):
    rng = np.random.default_rng(dims[0])
    lat = build_lattice(*dims)
    w = torch.from_numpy(_costs(lat, kind, rng)).cuda()
    count = 64 if dims[2] < 18 else 40
    box, src, dst = random_boxes(lat, count, seed=dims[1], lo=lo, hi=dims)
    dst[::9] = src[::9]
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()  # noqa: E731
    dg = DeviceGraph.from_lattice(lat)
    got = []
    for plan in (None, [{"max_nodes": 1 << 40, "impl": 0}]):
        dg.set_batch_plan(plan)
        got.append([a.cpu().numpy() for a in dg.batch_bbox(w, t(src), t(dst), t(box), path_cap=8192)])
    (n0, e0, l0), (n1, e1, l1) = got
    assert np.array_equal(l0, l1)
    for k in range(count):
        n = max(int(l0[k]), 0)
        assert np.array_equal(n0[k, :n], n1[k, :n]), k
        assert np.array_equal(e0[k, :max(n - 1, 0)], e1[k, :max(n - 1, 0)]), k
