"""Batched box searches without a plan against the same searches with one CTA
per search (a plan of impl 0 for every box), over the forms that the call
takes: box counts on both sides of the owner schedule's tile limit, boxes of one
cell, one layer and one row, layers around the depth up to which they are
swept, endpoints equal, unreachable and outside their box, integer costs (ties),
blocked and NaN edges, rows too short for the path, an explicit order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200.lattice import build_lattice, random_boxes, uniform_weights  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402


def _run(dg, w, src, dst, box, plan, cap, order=None):
    dg.set_batch_plan(plan)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).cuda()  # noqa: E731
    n, e, l = dg.batch_bbox(w, t(src), t(dst), t(box), order=None if order is None else t(order), path_cap=cap)
    return n.cpu().numpy(), e.cpu().numpy(), l.cpu().numpy()


@pytest.mark.parametrize("dims,count,lo", [
    ((60, 50, 6), 3, (1, 1, 1)), ((60, 50, 6), 300, (1, 1, 1)), ((90, 80, 18), 40, (8, 8, 18)),
    ((40, 40, 20), 30, (8, 8, 17)), ((300, 280, 5), 120, (100, 100, 4)), ((33, 17, 3), 50, (2, 2, 1)),
])
@pytest.mark.parametrize("costs", ["fractional", "integer"])
@pytest.mark.parametrize("cap", [1024, 24])
def test_default_equals_one_cta_per_search(dims, count, lo, costs, cap):
    lat = build_lattice(*dims)
    rng = np.random.default_rng(count + dims[0])
    w = uniform_weights(lat, seed=count, blocked_frac=0.1)
    if costs == "integer":
        w = np.where(np.isinf(w), w, rng.integers(0, 3, lat.E)).astype(np.float32)
    w[rng.choice(lat.E, lat.E // 50, replace=False)] = np.nan
    box, src, dst = random_boxes(lat, count, seed=count, lo=lo, hi=dims)
    dst[::7] = src[::7]
    src[3::11] = rng.integers(0, lat.N, len(src[3::11]))  # mostly outside their boxes
    dst[5::13] = rng.integers(0, lat.N, len(dst[5::13]))
    dg = DeviceGraph.from_lattice(lat)
    wt = torch.from_numpy(w).cuda()
    one = [{"max_nodes": 1 << 40, "impl": 0}]
    order = rng.permutation(count)
    a, b = _run(dg, wt, src, dst, box, None, cap, order), _run(dg, wt, src, dst, box, one, cap)
    assert np.array_equal(a[2], b[2])
    for k in range(count):
        n = max(int(a[2][k]), 0)
        assert np.array_equal(a[0][k, :n], b[0][k, :n]), k
        assert np.array_equal(a[1][k, :max(n - 1, 0)], b[1][k, :max(n - 1, 0)]), k
