"""The batch workspace's layout holds nothing that no kernel reads or writes."""
import ctypes

from dsplat import _native as N


def test_no_room_for_tile_counts_per_point():
    v = (N.View * 16)()
    for k in range(16):
        v[k].width, v[k].height = 640, 480
    n = 1 << 20
    L = N.BatchLayout()
    assert N.lib().dsplat_gauss_batch_layout(n, 16, v, 8, 0, 1 << 24, ctypes.byref(L)) == 0
    spans_and_sorted_spans = 2 * 8 * 16 * n + 1024
    assert L.off_order - L.off_rect <= spans_and_sorted_spans + 4 * 16 * n  # and the depth keys
