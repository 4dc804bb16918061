"""The routing loop with the searches' weights gathered once per call and kept by
the commits (boxes of the call hold as many cells as the lattice) against one
call per net, whose searches gather their own: paths, usage and costs, over two
passes (the second rips up), in the caller's order and in groups of disjoint
boxes, and on a lattice with column vias, which always gathers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200 import _lib  # noqa: E402
from orthoroute_b200._lib import check, ptr  # noqa: E402
from orthoroute_b200.accounting import DeviceEdgeAccountant  # noqa: E402
from orthoroute_b200.lattice import bbox_with_margin, build_lattice  # noqa: E402
from orthoroute_b200.negotiate import level_groups, level_schedule  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402


@pytest.mark.parametrize("dims,kw", [((64, 48, 4), {}), ((37, 50, 7), {}), ((30, 1, 3), {}),
                                     ((40, 36, 5), dict(planar="inner", vias="full", duplicate_vias=True))])
@pytest.mark.parametrize("levels", [False, True])
def test_kept_weights_equal_gathered_ones(dims, kw, levels):
    lat = build_lattice(*dims, **kw)
    rng = np.random.default_rng(dims[0])
    M, cap = 60, 512
    pins = rng.integers(0, dims[0] * dims[1], (2, M)).astype(np.int32)
    src, dst = np.ascontiguousarray(pins[0]), np.ascontiguousarray(pins[1])
    boxes = np.ascontiguousarray(bbox_with_margin(lat, src, dst, 3), dtype=np.int32)
    v = (boxes[:, 1] - boxes[:, 0] + 1) * (boxes[:, 3] - boxes[:, 2] + 1) * (boxes[:, 5] - boxes[:, 4] + 1)
    assert v.sum() >= lat.N  # one call keeps the weights
    order, groups = np.arange(M, dtype=np.int32), None
    if levels:
        order, groups = level_groups(order, level_schedule(boxes))
    dg = DeviceGraph.from_lattice(lat)
    base = torch.from_numpy(lat.base_cost).cuda().float()

    def run(calls):
        acc = DeviceEdgeAccountant(lat.E)
        cost = base.clone()
        nodes = torch.zeros((M, cap), dtype=torch.int32, device="cuda")
        edges = torch.full((M, cap), -1, dtype=torch.int32, device="cuda")
        lens = torch.zeros(M, dtype=torch.int32, device="cuda")
        for _ in range(2):
            for o, gp in calls:
                o = np.ascontiguousarray(o, dtype=np.int32)
                gp = None if gp is None else np.ascontiguousarray(gp, dtype=np.int32)
                check(_lib.load().orsp_route_nets(
                    dg.handle, M, ptr(src), ptr(dst), ptr(boxes), int(o.size), ptr(o),
                    0 if gp is None else int(gp.size - 1), ptr(gp), ptr(nodes), ptr(edges), cap, ptr(lens), ptr(cost),
                    ptr(base), ptr(acc.usage), ptr(acc.present), ptr(acc.capacity), ptr(acc.history), 0.5, 1.0, 1.0,
                    1.0, 1, 0), "orsp_route_nets")
        torch.cuda.synchronize()
        ln = lens.cpu().numpy()
        n, e = nodes.cpu().numpy(), edges.cpu().numpy()
        return (ln, [n[k, :ln[k]] for k in range(M)], [e[k, :max(ln[k] - 1, 0)] for k in range(M)],
                acc.usage.cpu().numpy(), cost.cpu().numpy().view(np.uint32))

    # one net per call: v < lat.N for all but the largest boxes
    one, each = run([(order, groups)]), run([([k], None) for k in order])
    assert (v < lat.N).any() and (one[0] > 1).any()
    assert np.array_equal(one[0], each[0])
    for k in range(M):
        assert np.array_equal(one[1][k], each[1][k]) and np.array_equal(one[2][k], each[2][k]), k
    assert np.array_equal(one[3], each[3]) and np.array_equal(one[4], each[4])
