"""One-dimensional problems, several steps per launch in registers: equal to the path of
one launch per stage bit for bit, over lengths at the edges of a 128-point segment,
step counts around a launch's, both boundary kinds, options, passes and types; a
cyclic problem whose ends differ does not take it."""
import numpy as np
import pytest

from libmpdataxx_b200 import opts as o
from test_gpu_parity import make_run

pytestmark = pytest.mark.gpu

OPTS = [(0, 1), (0, 2), (0, 3), (o.iga, 2), (o.fct, 2), (o.iga | o.fct, 2), (o.fct, 3), (o.tot, 3), (o.iga | o.tot | o.fct, 2),
        (o.tot | o.fct, 3)]


@pytest.mark.parametrize("bc", ["cyclic", "open"])
@pytest.mark.parametrize("opts,iters", OPTS)
@pytest.mark.parametrize("n,dtype,n_eqns,uff", [(5, np.float64, 1, 0), (33, np.float64, 2, 0), (128, np.float32, 1, 0),
                                                (129, np.float64, 5, 3), (1000, np.float32, 1, 0), (40001, np.float64, 1, 0)])
def test_line_equals_stages(n, dtype, n_eqns, uff, opts, iters, bc):
    rng = np.random.default_rng(n + iters)
    psi = [rng.uniform(0.5, 2.0, n).astype(dtype) for _ in range(n_eqns)]
    c = rng.uniform(-0.4, 0.4, n).astype(dtype)  # view element a: face a - 1 (+ 1/2)
    if bc == "cyclic":
        for a in psi:
            a[-1] = a[0]
    runs = []
    for path in ("general", "auto"):
        r = make_run((n,), opts, n_iters=iters, n_eqns=n_eqns, dtype=dtype, bcs=[bc] * 2, path=path, upwind_filter_freq=uff)
        for e, a in enumerate(psi):
            r.set_advectee(a, e)
        r.set_advector(c, 0)
        runs.append(r)
    for steps in (1, 23, 24, 26):
        for r in runs:
            r.advance(steps)
        for e in range(n_eqns):
            got = np.asarray(runs[1].advectee(e))
            assert np.isfinite(got).all()
            np.testing.assert_array_equal(got, runs[0].advectee(e))


def test_line_needs_consistent_seams():
    rng = np.random.default_rng(1)
    psi, runs = rng.uniform(0.5, 2.0, 50), []
    for path in ("general", "auto"):
        r = make_run((50,), o.iga | o.fct, bcs=["cyclic"] * 2, path=path)
        r.set_advectee(psi)
        r.set_advector(np.full(50, 0.3), 0)
        r.advance(30)
        runs.append(np.array(r.advectee()))
    np.testing.assert_array_equal(*runs)
