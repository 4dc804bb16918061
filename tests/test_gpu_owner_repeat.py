"""One search repeated many times under each schedule whose CTAs exchange
boundary values: every launch settles every node alike, bit for bit as the
oracle (an order of stores and messages that is not kept shows as distances that
are too large now and then)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200 import _lib  # noqa: E402
from orthoroute_b200.lattice import build_lattice, uniform_weights  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

import oracle as O  # noqa: E402


@pytest.mark.parametrize("dims", [(150, 150, 4), (270, 260, 3), (400, 330, 3)])
def test_repeated_searches_settle_alike(dims):
    lat = build_lattice(*dims)
    w = uniform_weights(lat, seed=11, blocked_frac=0.05)
    dg, wt = DeviceGraph.from_lattice(lat), torch.from_numpy(w).cuda()
    src = lat.N // 2 + 5
    _, ref, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [src])
    want = torch.from_numpy(ref.view(np.int32).copy()).cuda()
    dist = torch.empty(lat.N, dtype=torch.float32, device="cuda")
    for _ in range(200):
        assert dg.sssp(wt, src, -1, dist_out=dist)[0] == _lib.ORSP_OK
        assert torch.equal(dist.view(torch.int32), want)
