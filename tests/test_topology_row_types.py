"""A topology plan's row values are taken as int() and float() take them, whatever
their types, and refused where those refuse them: a missing sample is an error, not
NaN, a source of text has to be a whole number, and no value goes through a
rounding that int() does not make."""
from decimal import Decimal
from fractions import Fraction

import numpy as np
import pytest

import rustscan_b200 as G
from rustscan_b200 import _lib


def _row_by_row(rows):
    recs = (_lib.gsr_topo_row * max(len(rows), 1))()
    for i, (src, kind, sample) in enumerate(rows):
        recs[i] = _lib.gsr_topo_row(int(src), int(kind), float(sample), 0)
    return np.frombuffer(recs, G._TOPO_ROW, len(rows))


FILL = [(i % 7, i % 3, i / 8.0) for i in range(1500)]  # more rows than are packed at a time


@pytest.mark.parametrize("row", [(0, 0, None), (None, 0, 0.0), ("5.7", "1", "0.5"), ("1e3", 0, 0.0), (0, "0.0", 0.0),
                                 (0, 0, ""), (0, 0, 1j), ((1,), 0, 0.0), (0, 0, [1.0])])
def test_refused_as_row_by_row(row):
    for rows in ([row], FILL + [row], [row] + FILL):
        with pytest.raises(Exception) as want:
            _row_by_row(rows)
        with pytest.raises(want.type):
            G._plan_rows(rows)


@pytest.mark.parametrize("row", [(Decimal("0.99999999999999999999"), 0, 1.0), (Fraction(2 ** 60 - 1, 2 ** 60), 1, 1.0),
                                 (2, Decimal("1.9"), Decimal("0.1")), ("7", "1", "2.5"), (" 5 ", "1_0", "nan"),
                                 (b"5", 0, b"0.5"), (3.9, -0.5, 7), (-1, -2 ** 31, -0.0), (2 ** 32, 2 ** 31, 1e39),
                                 (2 ** 70, 0, float("inf")), (np.uint64(2 ** 63), np.int8(1), np.float16(0.1)),
                                 (True, False, True), (np.array(4), np.array([2]), np.array(0.25)),
                                 (1, 2, 1e-45), (1, 2, 16777217)])
@pytest.mark.filterwarnings("ignore:Conversion of an array")
def test_taken_as_row_by_row(row):
    for rows in ([row], FILL + [row], [row] + FILL, FILL[:1024], FILL[:1023] + [row], tuple(FILL) + (row,)):
        assert G._plan_rows(rows).tobytes() == _row_by_row(rows).tobytes()
