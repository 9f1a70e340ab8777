"""The explain table's break-even call against the costs measured on B200 (72,000
SVs, l = 11, d = 3: 10.8 ms for the table, 39.3 ns a window without it)."""

from gkmsvm_lite_b200 import explain


def test_break_even_call():
    windows = explain._TABLE_BUILD_S_PER_ENTRY * 4**11 * 11 / explain._DIRECT_S_PER_WINDOW
    assert abs(windows / (10.8e-3 / 39.3e-9) - 1) < 0.05
    assert abs(explain._TABLE_BUILD_S_PER_ENTRY * 4**11 * 11 / 10.8e-3 - 1) < 0.05
