"""Walks on either side of the largest boxes whose parents the search records
(200 KB for the walk: 88 tiles of 17 or 18 layers, 266 of 5 or 6): the same
paths as the walk on distances, which the same search with distances asked for
takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200.lattice import build_lattice, uniform_weights  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402


@pytest.mark.parametrize("tiles,nz", [((8, 11), 18), ((9, 10), 18), ((8, 11), 17), ((14, 19), 5), ((3, 89), 5),
                                      ((14, 19), 6), ((3, 89), 6)])
def test_paths_around_the_limit_of_recorded_parents(tiles, nz):
    dims = (16 * tiles[0], 16 * tiles[1], nz)
    lat = build_lattice(*dims)
    w = torch.from_numpy(uniform_weights(lat, seed=sum(dims), blocked_frac=0.03)).cuda()
    dg = DeviceGraph.from_lattice(lat)
    dist = torch.empty(lat.N, dtype=torch.float32, device="cuda")
    box = np.array([0, dims[0] - 1, 0, dims[1] - 1, 0, nz - 1])
    rng = np.random.default_rng(nz)
    for k in range(6):
        s, d = (int(v) for v in rng.integers(0, lat.N, 2))
        if k == 0:
            s, d = 0, lat.N - 1
        (st1, p1, _), (st2, p2, _) = (dg.sssp_box(w, s, d, box, dist_out=out, path_cap=8192) for out in (None, dist))
        assert st1 == st2 and (p1 is None) == (p2 is None)
        assert p1 is None or np.array_equal(p1.cpu().numpy(), p2.cpu().numpy())
