"""pd_cancel, whatever state its ticket is in."""
import time

import numpy as np
import pytest

from pripps_b200 import _lib, workloads
from pripps_b200.debye import solve
from pripps_b200.errors import DeviceError
from pripps_b200.serving import Server

pytestmark = pytest.mark.gpu


def _finished(srv, ticket):
    end = time.monotonic() + 60.0
    while not srv.poll(ticket):
        assert time.monotonic() < end
        time.sleep(1e-3)


def test_cancel_of_a_finished_request(gpu_ctx):
    """Not taken: the result is gone, for wait and poll. Taken: nothing changes."""
    req = workloads.small_globule(500, 4, nq=40).request
    want = solve(req, gpu_ctx)
    srv = Server(gpu_ctx)
    t = srv.submit(req)
    _finished(srv, t)
    srv.cancel(t)
    for call in (srv.wait, srv.poll):
        with pytest.raises(DeviceError) as e:
            call(t)
        assert e.value.code == _lib.PD_ECANCELED
    t = srv.submit(req)
    assert np.array_equal(srv.wait(t, timeout_s=60), want)
    srv.cancel(t)
    assert srv.poll(t)


def test_cancel_at_once_and_twice(gpu_ctx):
    srv = Server(gpu_ctx)
    t = srv.submit(workloads.small_globule(2000, 4, nq=200).request)
    srv.cancel(t)
    srv.cancel(t)
    with pytest.raises(DeviceError) as e:
        srv.wait(t, timeout_s=60)
    assert e.value.code == _lib.PD_ECANCELED
