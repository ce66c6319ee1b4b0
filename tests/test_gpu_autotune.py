"""The autotuner times the pair kernels, also on requests that a solve sums as
directions."""
import ctypes as C

import numpy as np
import pytest

from pripps_b200 import _lib, workloads

pytestmark = pytest.mark.gpu


def _execution_ms(ctx, req):
    """Device time of a plan's execution, and the form that ran."""
    import torch
    lib, r, p = _lib.lib(), req.c_struct(), C.c_void_p()
    _lib.check(lib.pd_plan_create(ctx.handle, C.byref(r), C.byref(p)), ctx.handle)
    xyz = torch.from_numpy(np.ascontiguousarray(req.xyz)).cuda()
    out = torch.empty((6, req.nq), dtype=torch.float64, device="cuda")
    s = torch.cuda.current_stream()
    best = 1e9
    for _ in range(8):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        _lib.check(lib.pd_plan_execute(ctx.handle, p, xyz.data_ptr(), out.data_ptr(),
                                       s.cuda_stream), ctx.handle)
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    form, mom = C.c_uint32(), C.c_uint32()
    _lib.check(lib.pd_plan_forms(ctx.handle, p, C.byref(form), C.byref(mom)), ctx.handle)
    lib.pd_plan_destroy(ctx.handle, p)
    return best, form.value


def test_autotuner_times_the_pair_kernels():
    req = workloads.small_globule(16_000, 5, nq=300, qmax=0.5, solvent=False,
                                  precision="fp32").request
    lib, r = _lib.lib(), req.c_struct()
    ctx = _lib.Context(0)
    try:
        t_dir, form = _execution_ms(ctx, req)
        assert form == 2
        k, tj, np_, ms = C.c_uint32(), C.c_uint32(), C.c_uint32(), C.c_double()
        _lib.check(lib.pd_autotune_request(ctx.handle, C.byref(r), C.byref(k), C.byref(tj),
                                           C.byref(np_), C.byref(ms)), ctx.handle)
        # a budget that leaves no room for the directions' arrays: the same request as pairs
        b = C.c_uint64()
        _lib.check(lib.pd_request_device_bytes(None, C.byref(r), 0, C.byref(b)), None)
        small = _lib.Context(0, mem_budget_bytes=b.value + b.value // 10)
        try:
            t_pairs, form = _execution_ms(small, req)
        finally:
            small.close()
        assert form != 2 and t_pairs > 2.0 * t_dir
        assert ms.value > 0.5 * t_pairs, (ms.value, t_pairs, t_dir)
    finally:
        ctx.close()
