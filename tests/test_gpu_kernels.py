"""Which kernels a run takes, and the fused kernels asked for by name.

On periodic grids the automatic path chooses between the fused kernel and the staged
step; stats()["path"] names the path whose conditions the fields met, stats()["kernels"]
the kernels that ran.  The fused kernels are run here with path="fused", whatever the
automatic path would choose at the size: FP64 against the oracle to 1e-12, FP32 to 1e-5
of the field's maximum, the bounds of the limiter exactly, bulk-tensor against
per-thread plane copies and every chunk length bit for bit.  In FP64 3D the staged step
gives the fused kernel's bits."""
import numpy as np
import pytest

from libmpdataxx_b200 import _lib, opts as o
from test_gpu_edges import NO_DIV, random_problem
from test_gpu_fused import CASES_2D, CASES_3D, periodic_setup, run_both
from test_gpu_parity import make_run, rel_err

pytestmark = pytest.mark.gpu
FORMULAS, STAGES, FUSED, LINE, BLOCK = (_lib.KERNELS_FORMULAS, _lib.KERNELS_STAGES, _lib.KERNELS_FUSED, _lib.KERNELS_LINE,
                                        _lib.KERNELS_BLOCK)
PATH_GENERAL, PATH_FUSED = _lib.PATH_GENERAL, _lib.PATH_FUSED
SMALL3, LARGE3 = (24, 22, 41), (130, 64, 130)  # 130 x 64 x 130: just above 10^6 points


@pytest.mark.parametrize("grid,opts,iters,dtype,path,kernels,reported", [
    (SMALL3, o.iga | o.fct, 2, np.float64, "auto", STAGES, PATH_FUSED),
    (LARGE3, o.iga | o.fct, 2, np.float64, "auto", STAGES, PATH_FUSED),
    (SMALL3, o.iga | o.fct, 2, np.float64, "fused", FUSED, PATH_FUSED),
    (SMALL3, o.iga | o.fct, 2, np.float32, "auto", STAGES, PATH_FUSED),
    (SMALL3, o.iga | o.fct, 2, np.float32, "fused", FUSED, PATH_FUSED),
    (LARGE3, o.iga | o.fct, 2, np.float32, "auto", FUSED, PATH_FUSED),
    ((40, 51), o.fct, 3, np.float64, "auto", STAGES, PATH_FUSED),
    ((40, 51), o.fct, 3, np.float32, "auto", FUSED, PATH_FUSED),
    ((40, 51), o.fct, 3, np.float64, "general", STAGES, PATH_GENERAL),
    ((40, 51), o.iga | o.tot, 2, np.float64, "auto", STAGES, PATH_GENERAL),
    ((40, 51), o.abs, 2, np.float64, "auto", FORMULAS, PATH_GENERAL)])
def test_kernels_taken(grid, opts, iters, dtype, path, kernels, reported):
    run, _ = run_both(periodic_setup(grid, seed=2), opts, iters, dtype, 0, path)
    assert run.stats()["kernels"] == _lib.KERNELS_NONE
    run.advance(1)
    st = run.stats()
    assert (st["kernels"], st["path"]) == (kernels, reported)


@pytest.mark.parametrize("n,opts,n_eqns,bc,kernels,reported", [
    (50, 0, 1, "cyclic", LINE, PATH_FUSED), (50, o.fct, 1, "cyclic", LINE, PATH_GENERAL), (50, 0, 2, "cyclic", LINE, PATH_GENERAL),
    (50, 0, 1, "open", LINE, PATH_GENERAL), (50, o.abs, 1, "cyclic", BLOCK, PATH_FUSED), (50, o.abs, 1, "open", FORMULAS, PATH_GENERAL)])
def test_kernels_taken_1d(n, opts, n_eqns, bc, kernels, reported):
    run = make_run((n,), opts, n_eqns=n_eqns, bcs=[bc] * 2, path="auto")
    for e in range(n_eqns):
        run.set_advectee(np.ones(n), e)
    run.set_advector(np.full(n, 0.3), 0)
    run.advance(1)
    st = run.stats()
    assert (st["kernels"], st["path"]) == (kernels, reported)


@pytest.mark.parametrize("grid,opts,iters", [(g, q, 2) for g, q in CASES_3D] + CASES_2D)
def test_fused_fp64_matches_oracle(grid, opts, iters):
    run, orc = run_both(periodic_setup(grid, seed=sum(grid) + iters), opts, iters, np.float64, 3, "fused")
    for chunk in (1, 2):
        run.advance(chunk)
        orc.advance(chunk)
        assert run.stats()["kernels"] == FUSED
        assert rel_err(np.array(run.advectee()), orc.advectee()) <= 1e-12


@pytest.mark.parametrize("grid,opts", CASES_3D + [(LARGE3, o.iga | o.fct)])
def test_staged_equals_fused_fp64_3d(grid, opts):
    s = periodic_setup(grid, seed=sum(grid))
    out = []
    for path, kernels in (("fused", FUSED), ("auto", STAGES)):
        run, _ = run_both(s, opts, 2, np.float64, 0, path)
        run.advance(3)
        assert run.stats()["kernels"] == kernels
        out.append(np.array(run.advectee()))
    np.testing.assert_array_equal(*out)


@pytest.mark.parametrize("path", ["fused", "auto"])
@pytest.mark.parametrize("grid,opts,iters", [((48, 40, 70), o.iga | o.fct, 2), ((19, 30, 70), o.iga, 2), ((21, 30, 70), o.fct, 2),
                                             ((60, 300), o.fct, 3), ((60, 300), o.fct, 2)])
def test_fp32_against_oracle_and_bounds(grid, opts, iters, path):
    s = periodic_setup(grid, seed=3)
    run, orc = run_both(s, opts, iters, np.float32, 10, path)
    run.advance(10)
    orc.advance(10)
    assert run.stats()["kernels"] == (STAGES if path == "auto" and len(grid) == 3 else FUSED)
    a, b = np.array(run.advectee(), np.float64), orc.advectee()
    assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
    if opts & o.fct:
        run.advance(15)
        psi = np.array(run.advectee())
        assert psi.min() >= np.float32(s["advectee"][0].min()) and psi.max() <= np.float32(s["advectee"][0].max())


@pytest.mark.parametrize("grid,opts", [((24, 120, 240), o.iga | o.fct), ((24, 120, 240), o.iga), ((70, 64, 130), o.iga | o.fct)])
def test_bulk_copies_bitwise(grid, opts):
    L, s, res = _lib.lib(), periodic_setup(grid, seed=17), {}
    try:
        for mode in (1, 0):
            L.mpdx_fused3d_bulk_copies(mode)
            run, orc = run_both(s, opts, 2, np.float32, 6, "fused")
            run.advance(6)
            assert run.stats()["kernels"] == FUSED
            res[mode] = np.array(run.advectee())
    finally:
        L.mpdx_fused3d_bulk_copies(1)
    np.testing.assert_array_equal(res[0], res[1])
    orc.advance(6)
    b = orc.advectee()
    assert np.abs(res[1].astype(np.float64) - b).max() <= 1e-5 * np.abs(b).max()


@pytest.mark.parametrize("grid,dtype,kernels", [(LARGE3, np.float64, FUSED), (LARGE3, np.float32, FUSED), (SMALL3, np.float64, FUSED),
                                                (SMALL3, np.float32, STAGES)])
def test_planes_setting(grid, dtype, kernels):
    """On the automatic path: taken by the handles that the header names, the same fields
    for every value, set before the run or between two advances."""
    L, s, res = _lib.lib(), periodic_setup(grid, seed=23), []
    try:
        for lx in (64, 8, 512):
            L.mpdx_fused3d_planes_per_cta(lx)
            run, _ = run_both(s, o.iga | o.fct, 2, dtype, 0)
            run.advance(4)
            assert run.stats()["kernels"] == kernels
            assert run.tuning3d()["chosen"] == (lx if kernels == FUSED else 0)
            res.append(np.array(run.advectee()))
        L.mpdx_fused3d_planes_per_cta(0)
        run, _ = run_both(s, o.iga | o.fct, 2, dtype, 0)
        run.advance(2)
        L.mpdx_fused3d_planes_per_cta(96)
        run.advance(2)
        res.append(np.array(run.advectee()))
        L.mpdx_fused3d_planes_per_cta(0)
        run, _ = run_both(s, o.iga | o.fct, 2, dtype, 0)
        run.advance(4)
        assert run.tuning3d()["chosen"] == 0
        res.append(np.array(run.advectee()))
    finally:
        L.mpdx_fused3d_planes_per_cta(0)
    for a in res[1:]:
        np.testing.assert_array_equal(a, res[0])


C, O, R = "cyclic", "open", "rigid"


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("opts,iters", [(0, 1), (0, 3), (o.fct, 2), (o.fct, 3), (o.iga, 2), (o.iga | o.fct, 3),
                                        (o.iga | o.tot | o.fct, 2), (o.tot, 3), (o.tot | o.fct, 3), (o.iga, 3), (o.iga | o.tot, 3),
                                        (o.iga | o.tot | o.fct, 3)])
@pytest.mark.parametrize("grid,bcs", [((37,), [C, C]), ((37,), [O, O]), ((9, 13), [C, C, O, O]), ((11, 12), [O, R, R, O]),
                                      ((70, 67), [R, R, C, C]), ((8, 9, 7), [C, C, O, O, R, R]), ((9, 7, 8), [R, O, C, C, O, O]),
                                      ((6, 21, 69), [O, O, O, O, O, O])])
def test_stages_equal_formulas(grid, bcs, opts, iters, dtype):
    """The staged step gives the bits of one kernel per formula.  The latter is reached by an
    option that changes nothing: in 1D and 3D fot, in 2D nug with its G of 1."""
    s, out = random_problem(grid, seed=sum(grid) + iters), []
    by_stages = not (iters == 3 and opts & o.iga and not opts & o.fct and R in bcs)  # the reference rewrites its velocity there
    for extra, kernels in ((0, STAGES if by_stages else FORMULAS), (o.nug if len(grid) == 2 else o.fot, FORMULAS)):
        run = make_run(grid, opts | extra, n_iters=iters, bcs=bcs, dtype=dtype, max_abs_div_eps=NO_DIV)
        run.set_advectee(s["advectee"][0].astype(dtype))
        for d, a in enumerate(s["advector"]):
            run.set_advector(a.astype(dtype), d)
        run.advance(3)
        assert run.stats()["kernels"] == kernels
        out.append(np.array(run.advectee()))
    np.testing.assert_array_equal(*out)
