"""The star lookup's window of bins around a direction, on the CPU.

The shading reads the stars of a row of bins as one run where the window lies
within the row.  The rule has to refuse every window that does not, the one of a
direction that is not finite included: its column converts to the most negative
int, and a run taken there would read outside the table."""
import ctypes as C
import os

import pytest

from blackhole_b200.build import CHECK_LIB, build_check

LON = 720
INT_MIN, INT_MAX = -(1 << 31), (1 << 31) - 1


@pytest.fixture(scope="module")
def window():
    if not os.path.exists(CHECK_LIB):
        build_check()
    return C.CDLL(CHECK_LIB).bhx_star_window


@pytest.mark.parametrize("half", [1, 2, 7, 100, 359, 360])
def test_only_a_window_within_the_row_is_one_run(window, half):
    bases = set(range(-LON, 2 * LON + 1)) | {INT_MIN, INT_MIN + 1, INT_MIN + half, INT_MIN + LON, INT_MAX,
                                             INT_MAX - half, INT_MAX - LON}
    for base in sorted(bases):
        assert window(base, half) == int(base - half >= 0 and base + half < LON), base
