"""The two forms of the GCR iteration on the device against the oracle: one cooperative
launch for the whole solve (one point per thread, and several), and two kernels per
inner step where the grid's axes are too long for the first form's table of index
rules (more than 2048 coordinates together).  Solutions agree to 1e-12 and the
iteration counts are equal, as for every FP64 pressure solve (both sides sum in
double-double, so the order of the sums does not show)."""
import numpy as np
import pytest

from runners import bq_oracle, bq_run
from test_gpu_boussinesq import random_bq

pytestmark = pytest.mark.gpu

CASES = [
    ((9, 7), ["cyclic"] * 4, 1),                             # one block
    ((9, 8, 7), ["cyclic"] * 4 + ["rigid"] * 2, 3),
    ((130, 33), ["cyclic"] * 2 + ["rigid"] * 2, 1),          # blocks of 128 threads, the last one partly used
    ((300, 254), ["cyclic"] * 4, 1),                         # 76200 points: just over one per thread
    ((45, 43, 41), ["rigid"] * 6, 2),                        # two points per pass, the second pass partly used
    ((2041, 9), ["cyclic"] * 2 + ["rigid"] * 2, 1),          # 2050 coordinates: two kernels per inner step
    ((2033, 8, 9), ["cyclic"] * 4 + ["rigid"] * 2, 1),
    ((2033, 8, 9), ["cyclic"] * 2 + ["rigid"] * 4, 4),
]


@pytest.mark.parametrize("grid,bcs,prs_k", CASES)
def test_gcr_forms_match_oracle(grid, bcs, prs_k):
    s = random_bq(grid, bcs, seed=sum(grid) + prs_k, prs_k=prs_k)
    run, orc = bq_run(s), bq_oracle(s)
    for _ in range(2):
        run.advance(1)
        orc.advance(1)
        for e in range(len(grid) + 1):
            got, want = np.asarray(run.advectee(e)), orc.advectee(e)
            assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
        assert run.stats()["gcr_iters"] == orc.last_iters
