"""Rounding error of the weight gradient against float64, on activations as a
ReLU leaves them.  The bounds are the errors of equal shares of the voxels per
CTA, each summed in one accumulator (relative L2, the smallest of three seeds):
longer sums than those, or sums of unequal length, are further off."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

from orthoroute_b200 import _lib  # noqa: E402
from orthoroute_b200._lib import ptr  # noqa: E402


@pytest.mark.parametrize("d,h,w,cin,cout,bound", [(18, 200, 200, 32, 32, 2.08e-6), (12, 184, 144, 32, 16, 8.06e-7),
                                                  (17, 112, 72, 16, 32, 3.70e-7), (11, 152, 136, 32, 32, 5.54e-7)])
def test_weight_gradient_error_is_that_of_even_sums(d, h, w, cin, cout, bound):
    g = torch.Generator(device="cuda").manual_seed(d + h + w)
    t = lambda c: torch.randn(d, h, w, c, generator=g, device="cuda")  # noqa: E731
    x, y, dy = torch.relu(t(cin)).to(torch.bfloat16), torch.relu(t(cout)).to(torch.bfloat16), t(cout).to(torch.bfloat16)
    dw = torch.zeros(27, cin, cout, device="cuda")
    assert _lib.load().orsp_warm_wgrad_tc(ptr(x), ptr(dy), ptr(y), ptr(dw), None, d, h, w, cin, cout, 0) == 0
    xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    gd = torch.where(y > 0, dy.double(), 0.0).reshape(-1, cout)
    want = torch.stack([xp[a:a + d, b:b + h, c:c + w].reshape(-1, cin).T @ gd
                        for a in range(3) for b in range(3) for c in range(3)])
    assert float((dw.double() - want).norm() / want.norm()) < bound
