"""The host check of the segmented layout on a window of 32 rows with more than
65,536 pieces (16-bit places cannot number them and are not read there)."""
import numpy as np

import multigraph_gb300 as mg


def test_window_of_more_pieces_than_places():
    n, rows, deg = 140_000, 32, 132_000
    row = np.zeros(n + 1, np.int32)
    row[1:rows + 1] = deg * (1 + np.arange(rows))
    row[rows + 1:] = rows * deg
    col = np.tile(np.arange(deg, dtype=np.int32), rows)
    assert mg.selftest_segmented_layout(row, col, threads=4) > 65_536
