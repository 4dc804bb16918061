"""Batched box searches with one CTA each, boxes above the shared-memory distance
array (24 K nodes) among them, which take the kernel's global-memory path: every
path and every edge list as the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200.lattice import build_lattice, random_boxes, uniform_weights  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

import oracle as O  # noqa: E402


@pytest.mark.parametrize("delta,ctas", [(0.75, 1), (2.0, 2)])
def test_one_cta_per_search_matches_oracle(delta, ctas):
    lat = build_lattice(90, 70, 6)
    w = uniform_weights(lat, seed=5, blocked_frac=0.03)
    dg = DeviceGraph.from_lattice(lat)
    dg.set_batch_plan([{"max_nodes": 1 << 40, "impl": 0, "delta": delta, "ctas_per_sm": ctas}])
    boxes, src, dst = random_boxes(lat, 60, seed=9, lo=(2, 2, 1), hi=(90, 70, 6))
    big = np.array([[0, 89, 0, 69, 0, 5], [3, 85, 1, 66, 0, 5], [0, 89, 10, 69, 0, 5]] * 4, np.int32)
    rng = np.random.default_rng(1)
    ends = [lat.node(rng.integers(3, 85, 12), rng.integers(10, 66, 12), rng.integers(0, 6, 12)) for _ in range(2)]
    boxes = np.concatenate([boxes, big]).astype(np.int32)
    src, dst = (np.concatenate([a, e]).astype(np.int32) for a, e in zip((src, dst), ends))
    nodes, edges, lens = dg.batch_bbox(*(torch.from_numpy(a).cuda() for a in (w, src, dst, boxes)), path_cap=2048)
    ref_nodes, ref_lens = O.batch_bbox(lat.indptr, lat.indices, w, lat.nx, lat.ny, lat.nz, src, dst, boxes, 2048)
    nodes, edges, lens = nodes.cpu().numpy(), edges.cpu().numpy(), lens.cpu().numpy()
    for k in range(len(src)):
        n = int(ref_lens[k])
        assert max(int(lens[k]), 0) * (n >= 2) == n * (n >= 2) and (lens[k] >= 2) == (n >= 2)
        if n >= 2:
            assert np.array_equal(nodes[k, :n], ref_nodes[k, :n])
            for u, v, e in zip(nodes[k, :n - 1], nodes[k, 1:n], edges[k]):
                assert lat.indptr[u] <= e < lat.indptr[u + 1] and lat.indices[e] == v
