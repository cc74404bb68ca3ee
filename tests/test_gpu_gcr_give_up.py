"""A wait of the one-launch pressure solve that runs out: the blocks leave, the call returns
MPDX_E_TIMEOUT, and the handle's next solves work (the arrival counter starts anew).  The
debug library has the entry point that takes an arrival away; every wait still ends, after
about two seconds."""
import pytest

from test_gpu_debug_paths import HEAD, debug_process

pytestmark = pytest.mark.gpu

SCRIPT = HEAD + r"""
L = _lib.lib()
L.mpdx_debug_lose_arrival.argtypes = [ctypes.c_void_p]
for grid, bcs, k in [((33, 29), [C, C, R, R], 1), ((45, 43, 41), [R] * 6, 2)]:
    s = random_bq(grid, bcs, seed=3, prs_k=k)
    run, ref = bq_run(s), bq_run(s)
    run._flush()
    assert L.mpdx_debug_lose_arrival(run.h) == 0
    codes = [L.mpdx_advance(run.h, 1)]
    message = L.mpdx_last_error(run.h).decode()
    # nothing was advanced: from the initial fields again, it gives an undisturbed handle's results
    for e, a in enumerate(s["advectee"]):
        run.set_advectee(a, e)
    codes.append(L.mpdx_advance(run.h, 2))
    ref.advance(2)
    err = max(rel(np.array(run.advectee(e)), np.array(ref.advectee(e))) for e in range(len(grid) + 1))
    out.append([codes, message, err, run.stats()["gcr_iters"] > 0])
print(json.dumps(out))
"""


def test_wait_that_runs_out():
    for codes, message, err, iterated in debug_process(SCRIPT):
        assert codes == [6, 0], (codes, message)  # MPDX_E_TIMEOUT, then MPDX_OK
        assert "gave up" in message
        assert iterated and err <= 1e-12, err
