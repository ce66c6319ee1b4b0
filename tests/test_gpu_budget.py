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


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mode", ["class", "weighted"])
def test_solve_in_exactly_its_smallest_layout(gpu_ctx, precision, mode):
    """With a budget of the bytes that pd_request_device_bytes names a solve runs, with
    one less it is refused; a batch too."""
    from pripps_b200.errors import DeviceError
    lib = _lib.lib()
    rng = np.random.default_rng(5)
    for n, nq, nf in ((700, 40, 1), (1500, 64, 1), (300, 50, 5)):
        xyz = rng.uniform(-14, 14, (nf, n, 3) if nf > 1 else (n, 3))
        w = rng.uniform(0, 2, n) if mode == "weighted" else np.where(rng.random(n) < 0.3, 1.25, 0.0)
        req = DebyeRequest(xyz, rng.integers(0, 3, n), rng.uniform(1, 8, (3, nq)), None, w,
                           rng.uniform(5, 10, nq), 0.0, 1.2, nq, None, precision)
        r, b = req.c_struct(), C.c_uint64()
        _lib.check(lib.pd_request_device_bytes(gpu_ctx.handle, C.byref(r), 1, C.byref(b)),
                   gpu_ctx.handle)
        want = solve(req, gpu_ctx)
        ctx = _lib.Context(0, mem_budget_bytes=b.value)
        try:
            err = term_errors(solve(req, ctx), want)
            assert np.all(err < (1e-5 if precision == "fp32" else 1e-10)), err
        finally:
            ctx.close()
        ctx = _lib.Context(0, mem_budget_bytes=b.value - 1)
        try:
            with pytest.raises(DeviceError):
                solve(req, ctx)
        finally:
            ctx.close()


def test_a_second_plan_takes_what_the_first_left(gpu_ctx):
    """A plan beside another in a budget that holds both as pairs only."""
    lib = _lib.lib()
    rng = np.random.default_rng(7)
    n, nq = 2500, 64
    req = DebyeRequest(rng.uniform(-16, 16, (n, 3)), rng.integers(0, 4, n),
                       rng.uniform(1, 8, (4, nq)), None, None, None, 0.0, 1.8, nq, None, "fp32")
    r, p, dbytes = req.c_struct(), C.c_void_p(), C.c_uint64()
    _lib.check(lib.pd_plan_create(gpu_ctx.handle, C.byref(r), C.byref(p)), gpu_ctx.handle)
    lib.pd_plan_info(p, None, None, None, None, C.byref(dbytes), None)
    lib.pd_plan_destroy(gpu_ctx.handle, p)
    ctx = _lib.Context(0, mem_budget_bytes=dbytes.value + _bytes(lib, r))
    try:
        plans = []
        for _ in range(2):
            plans.append(C.c_void_p())
            _lib.check(lib.pd_plan_create(ctx.handle, C.byref(r), C.byref(plans[-1])), ctx.handle)
        x, outs = np.ascontiguousarray(req.xyz), []
        for q in plans:
            outs.append(np.empty((6, nq)))
            _lib.check(lib.pd_plan_execute_host(ctx.handle, q, _lib.dptr(x), _lib.dptr(outs[-1])),
                       ctx.handle)
            lib.pd_plan_destroy(ctx.handle, q)
        assert np.all(term_errors(outs[1], outs[0]) < 1e-5)
    finally:
        ctx.close()
