"""Waits of the tensor-core convolutions and of the weight gradient that may not
wait (ORSP_WAIT_NS=0): every launch ends, and it gave up as a whole and the
status says so, or it is right (a single try of the hardware's wait can outlast
the whole wait); the next launch with the usual limit is right and reports
nothing.  The plane kernels with and without a mask, and the warp-specialised
kernel of wider layers."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200 import _lib  # noqa: E402
from orthoroute_b200._lib import ptr  # noqa: E402

D, H, W = 6, 40, 200


def _status():
    v = ctypes.c_int32(-1)
    assert _lib.load().orsp_warm_tc_status(ctypes.byref(v)) == 0
    return v.value


@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 32), (64, 32), (32, 64)])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("wgrad", [False, True])
def test_a_launch_that_may_not_wait_ends_and_says_so(cin, cout, masked, wgrad, monkeypatch):
    if wgrad and max(cin, cout) > 32:
        pytest.skip("one barrier per step, whose wait is voted by the block")
    lib = _lib.load()
    g = torch.Generator().manual_seed(cin + cout)
    t = lambda *s: torch.randn(*s, generator=g).cuda().to(torch.bfloat16)  # noqa: E731
    x, dy, m = t(D, H, W, cin), t(D, H, W, cout), t(D, H, W, cout if wgrad else cin) if masked else None
    wt, b = (0.1 * t(27, cin, cout).float()).to(torch.bfloat16), torch.randn(cout, generator=g).cuda()

    def call(reference=False):
        if wgrad:
            out = torch.zeros(27, cin, cout, device="cuda")
            fn = lib.orsp_warm_wgrad if reference else lib.orsp_warm_wgrad_tc
            assert fn(ptr(x), ptr(dy), ptr(m), ptr(out), None, D, H, W, cin, cout, 0) == 0
        else:
            out = torch.empty(D, H, W, cout, device="cuda")
            fn = lib.orsp_warm_conv3d if reference else lib.orsp_warm_conv3d_tc
            assert fn(ptr(x), ptr(m), ptr(wt), ptr(b), None, ptr(out), D, H, W, cin, cout, 0, 0) == 0
        torch.cuda.synchronize()
        return out

    want = call(reference=True)
    monkeypatch.setenv("ORSP_WAIT_NS", "0")
    for _ in range(8):
        out = call()
        if _status() == 0:
            assert float((out - want).norm() / want.norm()) < 1e-5
    monkeypatch.delenv("ORSP_WAIT_NS")
    assert float((call() - want).norm() / want.norm()) < 1e-5
    assert _status() == 0
