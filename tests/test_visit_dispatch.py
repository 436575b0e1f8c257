"""Which kernel a per-point FP32 visit takes: the one measured faster (no GPU needed: the rule
is host code).  Both give the same bits (test_gpu_tile_visits.py, test_gpu_parity.py)."""
import pytest

from tests import kernel_entries


@pytest.mark.parametrize("a,b,strips", [(16, 16, 0), (24, 20, 0), (32, 16, 1), (30, 32, 1), (40, 24, 1), (48, 16, 1), (64, 16, 0),
                                        (128, 16, 0), (128, 24, 0), (64, 64, 1), (32, 128, 1), (72, 56, 0),
                                        (96, 40, 0), (256, 16, 0), (128, 64, 0)])
def test_levels(a, b, strips):
    assert kernel_entries.load().entry_visit_cluster_beats_tiles(a, b, 70) == strips
