"""Device-buffer transfers are ordered after the work already issued to the legacy default
stream, and so after that of the streams which that stream waits for: a buffer that a
blocking stream or the legacy stream is still writing is read when it is complete, and one
that is still being read is not overwritten."""
import ctypes

import numpy as np
import pytest
import torch

from libmpdataxx_b200 import _lib, opts as o
from test_gpu_parity import make_run

pytestmark = pytest.mark.gpu


def blocking_stream():
    torch.cuda.init()
    torch.zeros(1, device="cuda")
    s = ctypes.c_void_p()
    assert ctypes.CDLL("libcudart.so.12").cudaStreamCreate(ctypes.byref(s)) == 0
    return s.value


@pytest.mark.parametrize("kind", ["legacy", "blocking"])
def test_transfers_wait_for_the_legacy_stream(kind):
    grid = (64, 65)
    run = make_run(grid, o.iga | o.fct)
    stream = torch.cuda.default_stream() if kind == "legacy" else torch.cuda.ExternalStream(blocking_stream())
    a, b = (torch.zeros(grid, dtype=torch.float64, device="cuda") for _ in range(2))
    b2 = torch.zeros_like(b)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(1 << 28)  # about 0.15 s
        a.fill_(3.0)
    run.set_field_device(_lib.FIELD_ADVECTEE, 0, a.data_ptr())
    np.testing.assert_array_equal(np.array(run.advectee()), 3.0)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(1 << 28)
        b2.copy_(b)  # reads b before the download below writes it
    run.get_field_device(_lib.FIELD_ADVECTEE, 0, b.data_ptr())
    torch.cuda.synchronize()
    assert (b2 == 0).all() and (b == 3).all()
