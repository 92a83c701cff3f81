"""Rectangle lists as callers give them: the table handed to the library, and
what is refused (SimulationEngine._rect_clips; no GPU needed)."""
from fractions import Fraction

import numpy as np
import pytest

import highuvlith_b200 as HB

TABLE = [[1.0, 2.0, 3.0, 4.0], [5.0, 6.0, 7.0, 8.5]]


def _table(clips):
    rects, offs = HB.SimulationEngine._rect_clips(clips, 1.0, 0.0)._keep
    assert rects.flags.c_contiguous and rects.dtype == np.float64 and offs.dtype == np.int32
    assert rects.shape == (offs[-1], 4)
    return rects.tolist(), offs.tolist()


@pytest.mark.parametrize("clip", [
    TABLE, [tuple(r) for r in TABLE], np.array(TABLE), np.array(TABLE, dtype=np.float32), np.array(TABLE).T.copy().T,
    [np.array(r) for r in TABLE], [[Fraction(v) for v in r] for r in TABLE], tuple(map(tuple, TABLE))])
def test_forms_of_one_table(clip):
    assert _table([clip, [], clip]) == (TABLE + TABLE, [0, 2, 2, 4])


def test_no_clips_and_empty_clips():
    assert _table([]) == ([], [0])
    assert _table([[], ()]) == ([], [0, 0, 0])


@pytest.mark.parametrize("clip,error", [
    ([((1.0, 2.0), (3.0, 4.0))], TypeError),               # nested pairs
    (np.zeros((2, 2, 2)), TypeError),
    ([1.0, 2.0, 3.0, 4.0], TypeError),                     # numbers in place of rectangles
    ([(None, 0.0, 1.0, 1.0)], TypeError),
    ([(1j, 0.0, 1.0, 1.0)], TypeError),
    ([(1.0, 2.0, 3.0)], ValueError),                       # too few numbers
    ([(1.0, 2.0), (3.0, 4.0)], ValueError),                # as many numbers as one rectangle has
    ([(1.0, 2.0, 3.0, 4.0, 5.0, 6.0, 7.0, 8.0)], ValueError)])
def test_refusals(clip, error):
    with pytest.raises(error):
        HB.SimulationEngine._rect_clips([TABLE, clip], 1.0, 0.0)
