"""The staged MPDATA step (one launch per stage, halo rules read in place) against the
oracle over the forms it accepts: 1 to 3 dimensions, boundary conditions mixed per
side, opts within fct, iga and tot, 1 to 3 passes, several equations per launch, the
upwind-only filter; FP64 to 1e-12 of the field's scale (the bound of the path it
replaces), FP32 to 1e-5.  Grids are ragged, small enough that most points are near a
face and, in one case, long enough for rows of several warps."""
import numpy as np
import pytest

from libmpdataxx_b200 import opts as o
from oracle import Oracle
from test_gpu_edges import NO_DIV, random_problem
from test_gpu_parity import make_run

pytestmark = pytest.mark.gpu

C, O, R = "cyclic", "open", "rigid"
OPTS = [(0, 1), (0, 3), (o.fct, 2), (o.fct, 3), (o.iga, 2), (o.iga | o.fct, 3), (o.iga | o.tot | o.fct, 2), (o.tot, 3),
        (o.tot | o.fct, 3)]
GRIDS = [((37,), [C, C]), ((37,), [O, O]), ((300,), [O, O]),
         ((9, 13), [C, C, O, O]), ((13, 9), [O, O, C, C]), ((11, 12), [O, R, R, O]), ((70, 67), [R, R, C, C]),
         ((8, 9, 7), [C, C, O, O, R, R]), ((7, 8, 9), [O, O, R, R, C, C]), ((9, 7, 8), [R, O, C, C, O, O]),
         ((6, 21, 69), [O, O, O, O, O, O])]


def check(grid, bcs, opts, iters, n_eqns=1, dtype=np.float64, steps=3, tol=1e-12, **kw):
    s = random_problem(grid, seed=sum(grid) + iters, n_eqns=n_eqns)
    run = make_run(grid, opts, n_iters=iters, n_eqns=n_eqns, bcs=bcs, dtype=dtype, max_abs_div_eps=NO_DIV, **kw)
    orc = Oracle(grid, opts, n_iters=iters, n_eqns=n_eqns, bcs=bcs, max_abs_div_eps=NO_DIV)
    if "upwind_filter_freq" in kw:
        orc.set_param("upwind_filter_freq", kw["upwind_filter_freq"])
    for e, a in enumerate(s["advectee"]):
        run.set_advectee(a.astype(dtype), e)
        orc.set_advectee(a.astype(dtype).astype(np.float64), e)
    for d, a in enumerate(s["advector"]):
        run.set_advector(a.astype(dtype), d)
        orc.set_advector(a.astype(dtype).astype(np.float64), d)
    run.advance(steps)
    orc.advance(steps)
    for e in range(n_eqns):
        want = orc.advectee(e)
        assert np.abs(np.asarray(run.advectee(e), np.float64) - want).max() <= tol * np.abs(want).max()


@pytest.mark.parametrize("opts,iters", OPTS)
@pytest.mark.parametrize("grid,bcs", GRIDS, ids=["x".join(map(str, g)) + "_" + "".join(b[0] for b in bc) for g, bc in GRIDS])
def test_stages_match_oracle(grid, bcs, opts, iters):
    if iters == 3 and "rigid" in bcs and len(grid) == 1:
        pytest.skip("rigid walls are for 2D and 3D")
    check(grid, bcs, opts, iters)


@pytest.mark.parametrize("grid,bcs", [((41,), [O, O]), ((12, 9), [O, O, C, C]), ((8, 9, 10), [C, C, R, R, O, O])])
def test_stages_equations_per_launch(grid, bcs):
    check(grid, bcs, o.iga | o.fct, 2, n_eqns=6)  # four equations in the first launch, two in the second


def test_stages_fp32():
    check((8, 9, 70), [C, C, O, O, O, O], o.iga | o.tot | o.fct, 2, dtype=np.float32, tol=1e-5)
