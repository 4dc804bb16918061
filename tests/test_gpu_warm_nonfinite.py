"""The weight gradient with infinities and NaN in its inputs, at the borders of
the grid and inside: they reach exactly the elements whose sum over the voxels
v of the grid, X[v + tap] (zero outside the grid) times G[v], holds them.
Against that sum in float64; its finite elements within the rounding of fp32
sums of random sign (1e-5 relative L2, as for finite inputs)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200 import _lib  # noqa: E402
from orthoroute_b200._lib import ptr  # noqa: E402

SIZES = [(3, 9, 33), (2, 16, 32), (5, 8, 70), (1, 1, 1)]
PLACES = [(0, 0, 0), (-1, -1, -1), (0, -1, 0), (-1, 0, -1), (0.5, 0.5, 0.5)]


def _want(x, g):
    d, h, w, _ = x.shape
    xp = torch.zeros(d + 2, h + 2, w + 2, x.shape[3], dtype=torch.float64)
    xp[1:-1, 1:-1, 1:-1] = x.double()
    taps = [(a, b, c) for a in range(3) for b in range(3) for c in range(3)]
    return torch.stack([(xp[a:a + d, b:b + h, c:c + w, :, None] * g.double()[..., None, :]).sum((0, 1, 2))
                        for a, b, c in taps])


@pytest.mark.parametrize("d,h,w", SIZES)
@pytest.mark.parametrize("cin,cout", [(32, 32), (16, 32), (32, 16)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("into", ["x", "dy"])
def test_non_finite_voxels_reach_their_own_taps(d, h, w, cin, cout, value, into):
    lib = _lib.load()
    gen = torch.Generator().manual_seed(d * 1000 + h * 100 + w + cin + cout)
    t = lambda *s: torch.randn(*s, generator=gen).to(torch.bfloat16)  # noqa: E731
    for place in PLACES:
        x, dy, yo = t(d, h, w, cin), t(d, h, w, cout), t(d, h, w, cout)
        at = tuple(int(p * n) if p >= 0 else n - 1 for p, n in zip(place, (d, h, w)))
        (x if into == "x" else dy)[at][3] = value
        for mask in (None, yo):
            g = dy if mask is None else torch.where(yo > 0, dy, torch.zeros_like(dy))
            want = _want(x, g)
            dw = torch.zeros(27, cin, cout, device="cuda")
            dev = [None if a is None else a.cuda() for a in (x, dy, mask)]
            assert lib.orsp_warm_wgrad_tc(*(ptr(a) for a in dev), ptr(dw), None, d, h, w, cin, cout, 0) == 0
            torch.cuda.synchronize()
            v = ctypes.c_int32(-1)
            assert lib.orsp_warm_tc_status(ctypes.byref(v)) == 0 and v.value == 0
            got, fin = dw.double().cpu(), torch.isfinite(want)
            assert torch.equal(torch.isnan(got), torch.isnan(want)), (place, mask is None)
            assert torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
            assert (got[fin] - want[fin]).norm() <= 1e-5 * want[fin].norm()
