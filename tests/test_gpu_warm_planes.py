"""The plane kernels of the convolution and of the weight gradient where their
tiles end: widths around the 30 (32) voxels of a patch row, heights around its
8 rows, one to many planes, every channel pair, with and without the ReLU
mask.  Against the WMMA kernels, which add the same bf16 products in fp32 in
another order: 27 x 32 terms of random sign leave about sqrt(864) x 2^-24 =
1.8e-6, bounded here by 1e-5 (relative L2)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200 import _lib  # noqa: E402
from orthoroute_b200._lib import ptr  # noqa: E402

SIZES = [(1, 1, 1), (1, 8, 30), (2, 9, 31), (3, 7, 29), (5, 17, 61), (19, 16, 33), (4, 40, 128), (18, 33, 200)]
CHANNELS = [(16, 16), (16, 32), (32, 16), (32, 32)]


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30))


def _data(d, h, w, cin, cout, masked):
    g = torch.Generator().manual_seed(d * 1000 + h * 100 + w + cin + cout)
    t = lambda *s: torch.randn(*s, generator=g).cuda().to(torch.bfloat16)  # noqa: E731
    return t(d, h, w, cin), t(d, h, w, cout), t(d, h, w, cin if masked == "x" else cout) if masked else None, g


def _no_expired_wait():
    v = ctypes.c_int32(-1)
    assert _lib.load().orsp_warm_tc_status(ctypes.byref(v)) == 0 and v.value == 0


@pytest.mark.parametrize("d,h,w", SIZES)
@pytest.mark.parametrize("cin,cout", CHANNELS)
@pytest.mark.parametrize("masked", ["", "x"])
def test_conv_planes(d, h, w, cin, cout, masked):
    lib = _lib.load()
    x, _, m, g = _data(d, h, w, cin, cout, masked)
    wt = (torch.randn(27, cin, cout, generator=g) * 0.1).cuda().to(torch.bfloat16)
    b = torch.randn(cout, generator=g).cuda()
    out = [torch.full((d, h, w, cout), float("nan"), device="cuda") for _ in range(2)]
    for fn, y in zip((lib.orsp_warm_conv3d_tc, lib.orsp_warm_conv3d), out):
        assert fn(ptr(x), ptr(m), ptr(wt), ptr(b), None, ptr(y), d, h, w, cin, cout, 0, 0) == 0
    torch.cuda.synchronize()
    _no_expired_wait()
    assert _rel(out[0], out[1]) < 1e-5


@pytest.mark.parametrize("d,h,w", SIZES)
@pytest.mark.parametrize("cin,cout", CHANNELS)
@pytest.mark.parametrize("masked", ["", "y"])
def test_wgrad_planes(d, h, w, cin, cout, masked):
    lib = _lib.load()
    x, dy, m, _ = _data(d, h, w, cin, cout, masked)
    out = [(torch.zeros(27, cin, cout, device="cuda"), torch.zeros(cout, device="cuda")) for _ in range(2)]
    for fn, (dw, db) in zip((lib.orsp_warm_wgrad_tc, lib.orsp_warm_wgrad), out):
        assert fn(ptr(x), ptr(dy), ptr(m), ptr(dw), ptr(db), d, h, w, cin, cout, 0) == 0
    torch.cuda.synchronize()
    _no_expired_wait()
    assert _rel(out[0][0], out[1][0]) < 1e-5
    assert _rel(out[0][1], out[1][1]) < 1e-5
