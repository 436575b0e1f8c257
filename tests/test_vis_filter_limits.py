"""Which levels take the one-launch viscosity filter: those where it was measured faster than
the loop graph (no GPU needed: the rule is host code)."""
import pytest

from tests import kernel_entries


# cells; faster in one launch: smoothing, with the ratio, both again on a stretched grid
@pytest.mark.parametrize("a,b,smooth,ratio,smooth_stretched,ratio_stretched", [
    (64, 16, 1, 1, 1, 1), (128, 32, 1, 1, 1, 1), (176, 44, 1, 1, 1, 0), (192, 48, 1, 0, 0, 0), (224, 56, 1, 0, 0, 0),
    (256, 64, 1, 0, 0, 0), (272, 68, 0, 0, 0, 0), (352, 88, 0, 0, 0, 0), (640, 160, 0, 0, 0, 0)])
def test_levels(a, b, smooth, ratio, smooth_stretched, ratio_stretched):
    f = kernel_entries.load().entry_vis_filter_fits
    assert (f(a, b, 0, 1), f(a, b, 0, 0)) == (smooth, ratio)
    assert (f(a, b, 1, 1), f(a, b, 1, 0)) == (smooth_stretched, ratio_stretched)
