"""A topology plan's rows as device records: the flat conversion equals the
row-by-row one, bit for bit, over everything the latter accepts, and refuses
what it refuses."""
import numpy as np
import pytest

import rustscan_b200 as G
from rustscan_b200 import _lib


def _row_by_row(rows):
    recs = (_lib.gsr_topo_row * max(len(rows), 1))()
    for i, (src, kind, sample) in enumerate(rows):
        recs[i] = _lib.gsr_topo_row(int(src), int(kind), float(sample), 0)
    return np.frombuffer(recs, G._TOPO_ROW, len(rows))


@pytest.mark.parametrize("rows", [
    [(0, 0, 0.0)],
    [(i * 7 % 1000, i % 3, i / 3.0) for i in range(5000)],
    [(-1, 0, 0.0), (2 ** 32 + 5, 1, 1e300), (3.9, -1.5, float("nan")), (np.int64(4), np.int32(2), np.float32(0.3)),
     (True, 0, 1), (2 ** 31, -5, -1e39)],
    [(2 ** 60 + 3, 0, 1.0), ("7", "1", "2.5")],
    [[1, 2, 3.5], np.array([4.0, 1.0, -0.0])],
])
def test_rows_equal_row_by_row(rows):
    assert G._plan_rows(rows).tobytes() == _row_by_row(rows).tobytes()


@pytest.mark.parametrize("rows", [[(1, 2)], [(1, 2, 3, 4)], [(1, 2), (1, 2, 3, 4)], [(float("nan"), 1, 1.0)],
                                  [(float("inf"), 1, 1.0)], [(1, 2, 3), 5], [(None, 1, 2.0)]])
def test_rows_refused_alike(rows):
    with pytest.raises(Exception) as want:
        _row_by_row(rows)
    with pytest.raises(want.type):
        G._plan_rows(rows)
