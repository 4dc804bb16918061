"""ROI expansion on bit sets against the oracle: rows that end inside, at and
just past a word, one-cell-wide lattices, 64 layers, the largest lattice that
fits and the first that does not (queues in shared memory, also one whose front
overflows them), waves that start side by side, on one node and at the borders."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle as O  # noqa: E402
from orthoroute_b200.lattice import build_lattice  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

REFERENCE = dict(planar="inner", vias="full", duplicate_vias=True)


@pytest.mark.parametrize("dims,kw", [
    ((31, 20, 5), {}), ((32, 20, 5), REFERENCE), ((33, 20, 4), REFERENCE), ((64, 7, 3), {}), ((65, 40, 6), REFERENCE),
    ((1, 40, 4), {}), ((70, 1, 4), {}), ((20, 20, 64), {}),
    ((220, 227, 6), REFERENCE),  # 9 534 words of at most 9 557
    ((225, 227, 6), REFERENCE),  # 10 896
    ((100, 100, 64), REFERENCE),
])
def test_bit_expansion_matches_oracle(dims, kw):
    lat = build_lattice(*dims, **kw)
    rng = np.random.default_rng(sum(dims))
    dg = DeviceGraph(lat.indptr, lat.indices, *dims)
    for k in range(8):
        s, d = (int(v) for v in rng.integers(0, lat.N, 2))
        if k == 0:
            d = s
        if k == 1:
            s, d = 0, lat.N - 1
        if k == 2:
            d = min(s + 1, lat.N - 1)
        depth = int(rng.choice([0, 1, 5, 30, 150]))
        max_nodes = int(rng.choice([1, 2, 50, max(1, lat.N // 3), lat.N + 10]))
        ref, ref_map = O.roi_bfs(lat.indptr, lat.indices, s, d, depth, max_nodes)
        roi, g2r = dg.roi_bfs(s, d, depth, max_nodes)
        assert np.array_equal(roi.cpu().numpy(), ref)
        assert np.array_equal(g2r.cpu().numpy(), ref_map)
        keep = rng.integers(0, lat.N, int(rng.integers(1, 12))).tolist() + [s]
        if len(ref) + len(keep) < lat.N:  # the output holds N entries
            ref, _ = O.roi_bfs(lat.indptr, lat.indices, s, d, depth, max_nodes, keep=keep)
            assert np.array_equal(dg.roi_bfs_keep(s, d, depth, max_nodes, keep).cpu().numpy(), ref)
