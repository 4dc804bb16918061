"""The plane convolution from two threads at a time, on layers of one kernel that
need different amounts of shared memory: every launch is accepted and right."""
import threading

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200 import _lib  # noqa: E402
from orthoroute_b200._lib import ptr  # noqa: E402


def test_layers_of_one_kernel_from_two_threads():
    lib, (d, h, w, cin) = _lib.load(), (2, 8, 30, 16)
    g = torch.Generator().manual_seed(3)
    x = torch.randn(d, h, w, cin, generator=g).cuda().to(torch.bfloat16)
    failed = []

    def work(cout):
        wt = torch.randn(27, cin, cout, generator=torch.Generator().manual_seed(cout)).cuda().to(torch.bfloat16)
        st = torch.cuda.Stream()
        out = [torch.empty(d, h, w, cout, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        args = lambda y: (ptr(x), None, ptr(wt), None, None, ptr(y), d, h, w, cin, cout, 0, st.cuda_stream)  # noqa: E731
        bad = lib.orsp_warm_conv3d(*args(out[0]))
        for _ in range(4000):
            bad = bad or lib.orsp_warm_conv3d_tc(*args(out[1]))
        st.synchronize()
        if bad or float((out[0] - out[1]).norm() / out[0].norm()) > 1e-5:
            failed.append((cout, bad))

    threads = [threading.Thread(target=work, args=(c,)) for c in (16, 32)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
