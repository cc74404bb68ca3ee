"""The staged step where a thread walks several planes along the first axis (from 1100
blocks of 128 positions on: 2, 4 or 8 planes, the last chunk shorter), against the oracle
at open, rigid and periodic sides: values carried from plane to plane, the short chunk
and the lists of faces spread over several rows of blocks.  Tolerances as for one plane
per thread."""
import numpy as np
import pytest

from libmpdataxx_b200 import opts as o
from test_gpu_stages import check

pytestmark = pytest.mark.gpu
C, O, R = "cyclic", "open", "rigid"

# grid: blocks across x chunks at the number of planes taken (and, one step up, too few)
TWO, FOUR, EIGHT = (23, 110, 120), (22, 150, 165), (19, 217, 217)  # 104 x 12 (6), 194 x 6 (3), 368 x 3
FLAT4, FLAT8 = (23, 24001), (45, 24001)                              # 188 x 6 (3), 188 x 6


@pytest.mark.parametrize("grid,bcs,opts,iters", [
    (TWO, [O, O, R, R, C, C], o.iga | o.fct, 2), (TWO, [C, C, O, O, R, R], o.tot | o.fct, 3),
    (FOUR, [R, R, C, C, O, O], o.fct, 2), (FOUR, [O, R, O, O, C, C], o.iga | o.tot | o.fct, 2),
    (EIGHT, [O, O, O, O, O, O], o.fct, 3), (EIGHT, [R, R, R, R, R, R], o.iga | o.fct, 2), (EIGHT, [C, C, C, C, C, C], o.tot, 2),
    (FLAT4, [O, O, C, C], o.iga | o.tot | o.fct, 2), (FLAT4, [C, C, R, O], o.fct, 3),
    (FLAT8, [R, R, O, O], o.fct, 2), (FLAT8, [O, R, R, O], o.iga | o.fct, 3), (FLAT8, [O, O, O, O], 0, 2)])
def test_walk_matches_oracle(grid, bcs, opts, iters):
    check(grid, bcs, opts, iters, steps=2)


def test_walk_fp32():
    check(EIGHT, [O, O, R, R, C, C], o.iga | o.tot | o.fct, 2, dtype=np.float32, steps=2, tol=1e-5)
