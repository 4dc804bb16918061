"""ROI expansion on uniform lattices against the oracle, where its forms end:
marks in shared memory and in global memory, a front that overflows its queue
(the general kernel then runs), lattices with missing edges (general kernel),
one-cell-wide lattices, lists at, above and below the node cap, and must-keep
nodes inside and outside the ROI."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle as O  # noqa: E402
from orthoroute_b200.lattice import build_lattice  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

REFERENCE = dict(planar="inner", vias="full", duplicate_vias=True)


def _without(lat, drop):
    """The CSR without the edges at positions `drop`."""
    keep = np.ones(lat.E, bool)
    keep[drop] = False
    ends = np.concatenate([[0], np.cumsum(keep)])
    return ends[lat.indptr].astype(np.int32), lat.indices[keep]


@pytest.mark.parametrize("dims,kw,missing", [
    ((5, 1, 4), {}, 0), ((1, 9, 3), {}, 0), ((33, 17, 3), {}, 0), ((64, 50, 6), REFERENCE, 0),
    ((400, 320, 6), {}, 0),            # marks in global memory
    ((60, 60, 64), REFERENCE, 0),      # front larger than its queue
    ((40, 40, 5), {}, 7), ((40, 30, 5), REFERENCE, 9),
])
def test_lattice_expansion_matches_oracle(dims, kw, missing):
    lat = build_lattice(*dims, **kw)
    rng = np.random.default_rng(sum(dims) + missing)
    indptr, indices = _without(lat, rng.choice(lat.E, missing, replace=False)) if missing else (lat.indptr, lat.indices)
    dg = DeviceGraph(indptr, indices, *dims)
    for k in range(10):
        s, d = (int(v) for v in rng.integers(0, lat.N, 2))
        if k == 0:
            d = s
        depth = int(rng.choice([0, 1, 5, 30, 150]))
        max_nodes = int(rng.choice([1, 2, 50, max(1, lat.N // 3), lat.N + 10]))
        ref, ref_map = O.roi_bfs(indptr, indices, s, d, depth, max_nodes)
        roi, g2r = dg.roi_bfs(s, d, depth, max_nodes)
        assert np.array_equal(roi.cpu().numpy(), ref)
        assert np.array_equal(g2r.cpu().numpy(), ref_map)
        keep = rng.integers(0, lat.N, int(rng.integers(1, 12))).tolist() + [s]
        keep += keep[:2]
        if len(ref) + len(keep) < lat.N:  # the output holds N entries
            ref, _ = O.roi_bfs(indptr, indices, s, d, depth, max_nodes, keep=keep)
            assert np.array_equal(dg.roi_bfs_keep(s, d, depth, max_nodes, keep).cpu().numpy(), ref)
