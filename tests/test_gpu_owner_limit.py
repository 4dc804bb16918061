"""Searches under the owner schedules that cannot end by themselves: costs whose
sum around a loop is negative lower distances without end.  With a short budget
(ORSP_BUDGET_NS) the launch ends as a timeout, busy tiles included, and the next
search on the same graph is right.  A search that does end may take the whole
budget, however short the limit of a single wait (ORSP_WAIT_NS).  One tile per
CTA, two per SM, and tiles that visiting owners take."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200 import _lib  # noqa: E402
from orthoroute_b200._lib import OrspError  # noqa: E402
from orthoroute_b200.lattice import build_lattice, uniform_weights  # noqa: E402
from orthoroute_b200.solver import DeviceGraph  # noqa: E402

import oracle as O  # noqa: E402


@pytest.mark.parametrize("dims", [(20, 30, 4), (100, 90, 18), (250, 240, 5), (330, 320, 3)])
@pytest.mark.parametrize("target", [False, True])
def test_a_search_without_end_is_a_timeout(dims, target, monkeypatch):
    lat = build_lattice(*dims)
    dg = DeviceGraph.from_lattice(lat)
    w = uniform_weights(lat, seed=5, blocked_frac=0.02)
    loop = np.where(np.isinf(w), w, np.float32(-0.001)).astype(np.float32)
    dst = lat.N - 3 if target else -1
    dist = torch.empty(lat.N, dtype=torch.float32, device="cuda")
    monkeypatch.setenv("ORSP_BUDGET_NS", "20000000")
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    with pytest.raises(OrspError) as e:
        dg.sssp(torch.from_numpy(loop).cuda(), 7, dst, dist_out=None if target else dist, path_cap=4096)
    assert e.value.status == _lib.ORSP_ERR_TIMEOUT
    assert time.perf_counter() - t0 < 2.0
    monkeypatch.delenv("ORSP_BUDGET_NS")
    assert dg.sssp(torch.from_numpy(w).cuda(), 7, -1, dist_out=dist)[0] == _lib.ORSP_OK
    _, ref, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [7])
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("dims", [(100, 90, 18), (250, 240, 5), (330, 320, 3)])
def test_the_budget_alone_limits_a_search(dims, monkeypatch):
    lat = build_lattice(*dims)
    w = uniform_weights(lat, seed=6, blocked_frac=0.02)
    dist = torch.empty(lat.N, dtype=torch.float32, device="cuda")
    monkeypatch.setenv("ORSP_WAIT_NS", "1")
    assert DeviceGraph.from_lattice(lat).sssp(torch.from_numpy(w).cuda(), 7, -1, dist_out=dist)[0] == _lib.ORSP_OK
    _, ref, _, _ = O.dijkstra(lat.indptr, lat.indices, w, [7])
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), ref.view(np.uint32))
