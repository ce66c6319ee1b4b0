"""Larger requests of a mixed burst leave the GPU to the small ones, in a loop that has
served bursts before as in a fresh one (where starting up gives the small ones time)."""
import threading

import numpy as np
import pytest

from pripps_b200 import _lib, workloads
from pripps_b200.debye import solve
from pripps_b200.serving import Server

pytestmark = pytest.mark.gpu


def _small(k, n_small):
    rng = np.random.default_rng(3)
    specs = [(int(rng.integers(300, 2500)), int(rng.integers(30, 400)), bool(k % 3))
             for k in range(n_small)]
    return [workloads.small_globule(n, 100 + k, nq=nq, solvent=sol).request
            for k, (n, nq, sol) in enumerate(specs)]


def test_bursts_after_each_other():
    """Six bursts of eighty small requests behind two of 25,000 atoms: most small ones
    are done before the large ones every time."""
    ctx = _lib.Context(0)
    try:
        small = _small(3, 80)
        big = [workloads.small_globule(25_000, 7 + k, nq=300).request for k in range(2)]
        srv = Server(ctx)
        for _ in range(6):
            tickets = [srv.submit(r) for r in big + small]
            for t in tickets:
                srv.wait(t, timeout_s=60)
            done_big = min(srv.times(t)[2] for t in tickets[:2])
            assert sum(srv.times(t)[2] < done_big for t in tickets[2:]) >= 60
    finally:
        ctx.close()


def test_a_larger_request_is_not_held_for_good():
    """Beside clients that keep small requests in flight a larger one is done, and is
    the same as alone."""
    ctx = _lib.Context(0)
    try:
        small = _small(5, 12)
        big = workloads.small_globule(12_000, 5, nq=400).request
        want = solve(big, ctx)
        srv, stop = Server(ctx), threading.Event()

        def client(k):
            while not stop.is_set():
                srv.wait(srv.submit(small[k % 12]), timeout_s=60)
                k += 1
        threads = [threading.Thread(target=client, args=(4 * k,)) for k in range(3)]
        for t in threads:
            t.start()
        try:
            for _ in range(5):
                assert np.array_equal(srv.wait(srv.submit(big), timeout_s=10), want)
        finally:
            stop.set()
            for t in threads:
                t.join()
    finally:
        ctx.close()
