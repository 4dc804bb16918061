"""Whole-array accounting updates at the lengths and alignments where their
four-edges-per-thread form ends: every remainder of four, and arrays that start
off a 16-byte boundary.  Bit for bit against the numpy restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

import oracle as O  # noqa: E402
from orthoroute_b200.accounting import DeviceEdgeAccountant  # noqa: E402


def _bits(a):
    return np.asarray(a, dtype=np.float32).view(np.uint32)


def _off(t, off):
    """The tensor's values in memory that starts `off` elements past an aligned address."""
    buf = torch.empty(t.numel() + off, dtype=t.dtype, device="cuda")
    buf[off:].copy_(t)
    return buf[off:]


@pytest.mark.parametrize("E", [1, 3, 4, 5, 1022, 1023, 4097, 148 * 32 * 256 * 4 + 7])
@pytest.mark.parametrize("off", [0, 1])
def test_updates_at_remainders_and_alignments(E, off):
    rng = np.random.default_rng(E + off)
    usage = rng.integers(0, 4, E).astype(np.int32)
    ema = (rng.random(E) * 3).astype(np.float32)
    hist = np.where(rng.random(E) < 0.3, rng.random(E) * 20, 0).astype(np.float32)
    base = rng.choice(np.array([1.0, 3.0], np.float32), size=E)
    kind = (rng.random(E) < 0.5).astype(np.uint8)
    layer = rng.integers(0, 7, E).astype(np.uint8)
    bias = np.array([0.0, 0.3, 0.5, 0.9, 1.0, 1.4, 2.0], np.float32)
    cap = np.ones(E, np.float32)
    dev = {k: _off(torch.from_numpy(v).cuda(), off) for k, v in
           {"usage": usage, "ema": ema, "hist": hist, "base": base, "kind": kind, "layer": layer, "cap": cap}.items()}
    acc = DeviceEdgeAccountant(E)
    acc.usage, acc.present_ema, acc.history, acc.capacity = dev["usage"], dev["ema"], dev["hist"], dev["cap"]
    acc.present = _off(torch.zeros(E, device="cuda"), off)
    acc.total_cost = _off(torch.zeros(E, device="cuda"), off)

    present = usage.astype(np.float32)
    acc.refresh_from_canonical()
    assert np.array_equal(acc.present.cpu().numpy(), present)
    assert acc.compute_overuse() == tuple(int(v) for v in O.compute_overuse(present, cap))
    ema_ref = O.update_present_ema(present, ema, 0.4)
    acc.update_present_ema(beta=0.4)
    assert np.array_equal(_bits(acc.present_ema.cpu().numpy()), _bits(ema_ref))
    for more, ref in (({}, {}), ({"edge_layer": dev["layer"], "layer_bias_per_layer": bias, "edge_kind": dev["kind"]},
                               {"edge_layer": layer, "layer_bias_per_layer": bias, "edge_kind": kind})):
        acc.update_costs(dev["base"], 1.125, 0.7, add_jitter=True, base_cost_weight=0.3, **more)
        want = O.update_costs(base, ema_ref, cap, hist, 1.125, 0.7, add_jitter=True, base_cost_weight=0.3, **ref)
        assert np.array_equal(_bits(acc.total_cost.cpu().numpy()), _bits(want))
    want = O.update_history(hist, present, cap, 1.25, base_costs=base, history_cap_multiplier=15.0)
    acc.update_history(1.25, base_costs=dev["base"], history_cap_multiplier=15.0, use_raw_present=True)
    assert np.array_equal(_bits(acc.history.cpu().numpy()), _bits(want))
