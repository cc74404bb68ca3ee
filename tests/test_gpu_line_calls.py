"""Calls on one-dimensional problems that the kernel of several steps per launch must
leave as they are: a first advance under stream capture, which has no room for
allocations, and an advance after an upload, which returns before the device is done."""
import time

import numpy as np
import pytest
import torch

from libmpdataxx_b200 import _lib, opts as o
from test_gpu_parity import make_run

pytestmark = pytest.mark.gpu


def pair(n, opts, n_eqns, iters=2, bc="cyclic", **kw):
    rng = np.random.default_rng(n + n_eqns)
    psi = [rng.uniform(0.5, 2.0, n) for _ in range(n_eqns)]
    for a in psi:
        a[-1] = a[0]
    runs = [make_run((n,), opts, n_iters=iters, n_eqns=n_eqns, bcs=[bc] * 2, path=p, **kw) for p in ("general", "auto")]
    for r in runs:
        for e, a in enumerate(psi):
            r.set_advectee(a, e)
        r.set_advector(np.full(n, 0.3), 0)
    return runs


@pytest.mark.parametrize("opts,n_eqns,iters,bc", [(o.iga | o.fct, 2, 2, "cyclic"), (o.fct, 5, 3, "cyclic"),
                                                  (o.iga | o.fct, 3, 2, "open"), (0, 2, 1, "cyclic")])
def test_first_advance_captured(opts, n_eqns, iters, bc):
    ref, run = pair(50, opts, n_eqns, iters, bc)
    ref.advance(2)
    s, g = torch.cuda.ExternalStream(run.stream), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        rc = run.L.mpdx_advance(run.h, 2)
    assert rc == _lib.MPDX_OK, run.L.mpdx_last_error(run.h).decode()
    with torch.cuda.stream(s):
        g.replay()
    run.sync()
    for e in range(n_eqns):
        np.testing.assert_array_equal(np.array(run.advectee(e)), ref.advectee(e))
    run.advance(3)  # eagerly, with the work arrays of all equations
    ref.advance(3)
    for e in range(n_eqns):
        np.testing.assert_array_equal(np.array(run.advectee(e)), ref.advectee(e))
    del g


@pytest.mark.parametrize("kind", ["sync", "async"])
def test_advance_after_upload_does_not_wait(kind):
    """The device is busy for about half a second when advance() is called."""
    ref, run = pair(3000, o.iga | o.fct, 1)
    for r in (ref, run):
        r.advance(2)
        r.sync()
    a = torch.from_numpy(np.array(ref.advectee())[::-1].copy()).pin_memory()
    if kind == "sync":
        run.set_advectee(a.numpy())
    else:
        run.set_field_async(_lib.FIELD_ADVECTEE, 0, a.data_ptr())
    with torch.cuda.stream(torch.cuda.ExternalStream(run.stream)):
        torch.cuda._sleep(1 << 30)
    t = time.perf_counter()
    assert run.L.mpdx_advance(run.h, 3) == _lib.MPDX_OK
    returned = time.perf_counter() - t
    run.sync()
    waited = time.perf_counter() - t
    assert waited > 0.3 and returned < 0.1 * waited, (returned, waited)
    ref.set_advectee(a.numpy())
    ref.advance(3)
    np.testing.assert_array_equal(np.array(run.advectee()), ref.advectee())
