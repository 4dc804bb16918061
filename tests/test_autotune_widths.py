"""Batch plans the autotuner times (no GPU): plans that sweep the same boxes are
one plan, timed once."""
import numpy as np

from orthoroute_b200.autotune import _sweep_widths


def test_a_second_tile_width_only_where_it_sweeps_other_boxes():
    assert _sweep_widths(np.array([1, 4, 16])) == (16,)
    assert _sweep_widths(np.array([17])) == (16,)
    assert _sweep_widths(np.array([4, 18])) == (16, 32)
    assert _sweep_widths(np.array([], np.int32)) == (16,)
