"""A velocity that changes between advances (the loop of a host model that uploads an
advector, advances and downloads).  On periodic grids every step must use the advector
that was set last, halos included: the same fields as a handle made anew for each step
(bit for bit) and as the fused kernels, which wrap their indices (FP64 3D bit for bit;
FP64 2D 1e-12 and FP32 1e-5 of the field's maximum, whose arithmetic differs in
rounding).  Uploads by the synchronous and asynchronous calls and from device memory,
and between the replays of a captured advance.  In 1D the halos are filled before the
first step only, as in the reference, on every path."""
import numpy as np
import pytest
import torch

from libmpdataxx_b200 import _lib, opts as o, setups
from test_gpu_parity import make_run

pytestmark = pytest.mark.gpu

CASES = [((24, 22, 41), o.iga | o.fct, 2, np.float64), ((9, 6, 5), o.fct, 2, np.float64), ((24, 22, 41), 0, 2, np.float64),
         ((24, 22, 41), o.iga | o.fct, 2, np.float32), ((40, 51), o.fct, 3, np.float64), ((33, 5), o.iga, 2, np.float64),
         ((40, 51), o.fct, 2, np.float32)]


def steps(grid, dtype, n=3):
    rng = np.random.default_rng(sum(grid))
    out = []
    for k in range(n):
        curl = setups.periodic_curl_3d(grid, 7 + k, cmax=0.4, dtype=np.float64) if len(grid) == 3 else \
            setups.periodic_curl_2d(grid[0], grid[1], 7 + k, cmax=0.4)
        psi = setups.wrap_periodic(rng.uniform(0.5, 2.0, size=tuple(g - 1 for g in grid)))
        out.append((np.ascontiguousarray(psi, dtype=dtype), [np.ascontiguousarray(a, dtype=dtype) for a in curl]))
    return out


def make(grid, opts, iters, dtype, path="auto"):
    return make_run(grid, opts, n_iters=iters, dtype=dtype, path=path, max_abs_div_eps=1e-4)


def upload(run, kind, idx, a, how, keep):
    if how == "host":
        run.set_field(kind, idx, a)
    elif how == "device":
        t = torch.from_numpy(a).cuda()
        keep.append(t)
        run.set_field_device(kind, idx, t.data_ptr())
    else:
        t = torch.from_numpy(a).pin_memory()
        keep.append(t)
        run.set_field_async(kind, idx, t.data_ptr())


@pytest.mark.parametrize("how", ["host", "device", "async"])
@pytest.mark.parametrize("grid,opts,iters,dtype", CASES)
def test_new_advector_each_step(grid, opts, iters, dtype, how):
    run, fused, keep = make(grid, opts, iters, dtype), make(grid, opts, iters, dtype, "fused"), []
    tol = 1e-5 if dtype == np.float32 else (0.0 if len(grid) == 3 else 1e-12)
    psi = steps(grid, dtype)[0][0]
    for r in (run, fused):
        r.set_advectee(psi)
    for _, adv in steps(grid, dtype):
        fresh = make(grid, opts, iters, dtype)
        fresh.set_advectee(np.array(run.advectee()))
        for d, a in enumerate(adv):
            upload(run, _lib.FIELD_ADVECTOR, d, a, how, keep)
            for r in (fused, fresh):
                r.set_advector(a, d)
        for r in (run, fused, fresh):
            r.advance(2)
        got, want = np.array(run.advectee()), np.array(fused.advectee())
        np.testing.assert_array_equal(got, fresh.advectee())
        assert np.abs(got - want).max() <= tol * np.abs(want).max()
        for ax in range(len(grid)):  # the last point of a periodic axis stays its first
            np.testing.assert_array_equal(got.take(-1, ax), got.take(0, ax))
        fused.set_advectee(got)
        fresh.close()


@pytest.mark.parametrize("grid,opts,iters,dtype", [CASES[0], CASES[3], CASES[4]])
def test_new_advector_between_replays(grid, opts, iters, dtype):
    run = make(grid, opts, iters, dtype)
    (psi, adv), (psi1, adv1) = steps(grid, dtype, 2)
    run.set_advectee(psi)
    for d, a in enumerate(adv):
        run.set_advector(a, d)
    run.advance(2)
    run.sync()
    s, g = torch.cuda.ExternalStream(run.stream), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        _lib.lib().mpdx_advance(run.h, 2)
    run.set_advectee(psi1)
    for d, a in enumerate(adv1):
        run.set_advector(a, d)
    with torch.cuda.stream(s):
        g.replay()
    run.sync()
    fresh = make(grid, opts, iters, dtype)
    fresh.set_advectee(psi1)
    for d, a in enumerate(adv1):
        fresh.set_advector(a, d)
    fresh.advance(2)
    np.testing.assert_array_equal(np.array(run.advectee()), fresh.advectee())
    # and eagerly after the capture
    run.set_advectee(psi)
    for d, a in enumerate(adv):
        run.set_advector(a, d)
    run.advance(1)
    fresh = make(grid, opts, iters, dtype)
    fresh.set_advectee(psi)
    for d, a in enumerate(adv):
        fresh.set_advector(a, d)
    fresh.advance(1)
    np.testing.assert_array_equal(np.array(run.advectee()), fresh.advectee())
    del g


@pytest.mark.parametrize("bc", ["cyclic", "open"])
@pytest.mark.parametrize("opts,n_eqns", [(0, 1), (o.iga | o.fct, 1), (o.fct, 2)])
def test_new_advector_1d_as_general(opts, n_eqns, bc):
    n, rng = 70, np.random.default_rng(4)
    psi = [rng.uniform(0.5, 2.0, n) for _ in range(n_eqns)]
    for a in psi:
        a[-1] = a[0]
    runs = [make_run((n,), opts, n_eqns=n_eqns, bcs=[bc] * 2, path=p) for p in ("general", "auto")]
    for k in range(3):
        c = rng.uniform(0.1, 0.4, n) if k else np.full(n, 0.3)
        for r in runs:
            for e, a in enumerate(psi):
                if k == 0:
                    r.set_advectee(a, e)
            r.set_advector(c, 0)
            r.advance(5)
        for e in range(n_eqns):
            np.testing.assert_array_equal(np.array(runs[1].advectee(e)), runs[0].advectee(e))
