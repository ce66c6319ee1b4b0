"""Memory budgets between what the pairs need and what the directions need on top."""
import ctypes as C

import numpy as np
import pytest

from conftest import term_errors
from pripps_b200 import _lib, workloads
from pripps_b200.debye import DebyeRequest, solve

pytestmark = pytest.mark.gpu


def _bytes(lib, r):
    b = C.c_uint64()
    _lib.check(lib.pd_request_device_bytes(None, C.byref(r), 0, C.byref(b)), None)
    return b.value


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_shards_of_a_plan_that_fits_as_pairs(gpu_ctx, precision):
    """The plan gave the directions up for the budget; so do its shards, which add up
    to the whole solve."""
    lib = _lib.lib()
    rng = np.random.default_rng(3)
    n, nq = 2500, 64
    xyz = rng.uniform(-16, 16, (n, 3))
    req = DebyeRequest(xyz, rng.integers(0, 4, n), rng.uniform(1, 8, (4, nq)), None,
                       rng.uniform(0, 2, n), rng.uniform(5, 10, nq), 0.0, 1.8, nq, None, precision)
    r = req.c_struct()
    whole = solve(req, gpu_ctx)
    p, dbytes = C.c_void_p(), C.c_uint64()
    _lib.check(lib.pd_plan_create(gpu_ctx.handle, C.byref(r), C.byref(p)), gpu_ctx.handle)
    lib.pd_plan_info(p, None, None, None, None, C.byref(dbytes), None)
    lib.pd_plan_destroy(gpu_ctx.handle, p)
    pairs = _bytes(lib, r)
    budget = pairs + (64 << 10)
    assert dbytes.value > 1.5 * budget  # the directions' arrays are what does not fit
    ctx = _lib.Context(0, mem_budget_bytes=budget)
    try:
        form, mom = C.c_uint32(), C.c_uint32()
        out = np.empty((6, nq))
        for world in (2, 3):
            total = np.zeros((6, nq))
            for rank in range(world):
                _lib.check(lib.pd_plan_create(ctx.handle, C.byref(r), C.byref(p)), ctx.handle)
                _lib.check(lib.pd_plan_set_shard(ctx.handle, p, rank, world), ctx.handle)
                lib.pd_plan_info(p, None, None, None, None, C.byref(dbytes), None)
                assert dbytes.value <= budget
                x = np.ascontiguousarray(req.xyz)
                _lib.check(lib.pd_plan_execute_host(ctx.handle, p, _lib.dptr(x), _lib.dptr(out)),
                           ctx.handle)
                _lib.check(lib.pd_plan_forms(ctx.handle, p, C.byref(form), C.byref(mom)),
                           ctx.handle)
                assert form.value != 2
                total += out
                lib.pd_plan_destroy(ctx.handle, p)
            err = term_errors(total, whole)
            assert np.all(err < (1e-5 if precision == "fp32" else 1e-10)), err
    finally:
        ctx.close()
