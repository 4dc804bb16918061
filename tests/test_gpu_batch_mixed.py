"""Batched boxes without a plan on a lattice deeper than the sweeps take: shallow
boxes beside deep ones, smaller and larger than the largest deep one, in one
launch with them or swept apart (by their number), all shallow, all deep, and one
of each.  Every path as the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200.lattice import build_lattice, uniform_weights  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

import oracle as O  # noqa: E402

DIMS = (30, 24, 22)


def _boxes(rng, n, side, depth):
    """n boxes of up to `side` cells in x and y and depths in `depth`, with ends inside."""
    lo, hi = [], []
    for _ in range(n):
        size = [int(rng.integers(1, min(side, d) + 1)) for d in DIMS[:2]] + [int(rng.integers(depth[0], depth[1] + 1))]
        a = [int(rng.integers(0, d - s + 1)) for d, s in zip(DIMS, size)]
        lo.append(a)
        hi.append([v + s - 1 for v, s in zip(a, size)])
    return np.array(lo), np.array(hi)


@pytest.mark.parametrize("shallow,deep", [((1, 30), (1, 6)), ((40, 30), (5, 8)), ((200, 6), (9, 30)), ((290, 8), (6, 20)),
                                          ((291, 8), (6, 20)), ((20, 12), (0, 1)), ((0, 1), (12, 20)), ((1, 1), (1, 1))])
def test_boxes_of_mixed_depth_match_oracle(shallow, deep):
    lat = build_lattice(*DIMS)
    w = uniform_weights(lat, seed=8, blocked_frac=0.03)
    rng = np.random.default_rng(shallow[0] + 10 * deep[0])
    parts = [_boxes(rng, *shallow, (1, 18)), _boxes(rng, *deep, (19, 22))]
    lo, hi = (np.concatenate([p[i].reshape(-1, 3) for p in parts]) for i in (0, 1))
    order = rng.permutation(len(lo))
    lo, hi = lo[order], hi[order]
    boxes = np.stack([lo, hi], 2).reshape(-1, 6).astype(np.int32)
    src, dst = (lat.node(*rng.integers(lo, hi + 1).T).astype(np.int32) for _ in range(2))
    dg = DeviceGraph.from_lattice(lat)
    nodes, edges, lens = dg.batch_bbox(*(torch.from_numpy(a).cuda() for a in (w, src, dst, boxes)), path_cap=512)
    ref_nodes, ref_lens = O.batch_bbox(lat.indptr, lat.indices, w, *DIMS, src, dst, boxes, 512)
    nodes, edges, lens = nodes.cpu().numpy(), edges.cpu().numpy(), lens.cpu().numpy()
    for k in range(len(src)):
        n = int(ref_lens[k])
        assert (lens[k] >= 2) == (n >= 2)
        if n >= 2:
            assert lens[k] == n and np.array_equal(nodes[k, :n], ref_nodes[k, :n])
            assert np.array_equal(lat.indices[edges[k, :n - 1]], nodes[k, 1:n])
