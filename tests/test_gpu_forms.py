"""Which form a frame's pairs are summed in (pd_plan_forms): the other tests hold
every form to the same tolerances, so only this one sees a rule that quietly
falls back to another form."""
import ctypes as C

import numpy as np
import pytest

from conftest import term_errors
from oracle import oracle as O
from pripps_b200 import _lib, synth
from pripps_b200.debye import DebyeRequest, solve

pytestmark = pytest.mark.gpu
GRID, MOMENTS, DIRECTIONS = 0, 1, 2
TOL = {"fp64": 1e-10, "fp32": 1e-5}


def _ball(n, radius, seed=1):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(n, 3))
    xyz = v / np.linalg.norm(v, axis=1)[:, None] * rng.random((n, 1)) ** (1 / 3)
    xyz -= xyz.mean(axis=0)
    return xyz * (radius / np.linalg.norm(xyz, axis=1).max())


def _globule(n, seed=1):
    r = synth.sphere_radius_for(n)
    return synth.rsa_points(n, (r, r, r), np.random.default_rng(seed))


def _rod(n, length, seed=1):
    rng = np.random.default_rng(seed)
    xy = rng.uniform(-1, 1, (4 * n, 2))
    xy = xy[(xy ** 2).sum(axis=1) < 1][:n] * 10.0
    return np.column_stack([xy, rng.uniform(-length / 2, length / 2, n)])


def _request(xyz, qmax, nq, precision, mode="vacuum", seed=2):
    rng = np.random.default_rng(seed)
    n = xyz.shape[-2]
    sp = rng.integers(0, 3, n)
    ff = rng.uniform(1, 8, (3, nq))
    if mode == "vacuum":
        return DebyeRequest(xyz, sp, ff, None, None, None, 0.0, qmax, nq, None, precision)
    return DebyeRequest(xyz, sp, ff, rng.uniform(0.2, 3, (3, nq)), rng.uniform(0, 2, n),
                        rng.uniform(5, 10, nq), 0.0, qmax, nq, None, precision)


def _run(ctx, req, shard=None):
    """Profiles of a plan's execution, and each frame's (form, moments)."""
    lib = _lib.lib()
    r, p = req.c_struct(), C.c_void_p()
    nf = req.xyz.shape[0] if req.xyz.ndim == 3 else 1
    form, mom = (C.c_uint32 * nf)(), (C.c_uint32 * nf)()
    out = np.empty((6, req.nq))
    _lib.check(lib.pd_plan_create(ctx.handle, C.byref(r), C.byref(p)), ctx.handle)
    try:
        assert lib.pd_plan_forms(ctx.handle, p, form, mom) == _lib.PD_EINVAL
        if shard:
            _lib.check(lib.pd_plan_set_shard(ctx.handle, p, *shard), ctx.handle)
        xyz = np.ascontiguousarray(req.xyz, dtype=np.float64)
        _lib.check(lib.pd_plan_execute_host(ctx.handle, p, _lib.dptr(xyz), _lib.dptr(out)),
                   ctx.handle)
        _lib.check(lib.pd_plan_forms(ctx.handle, p, form, mom), ctx.handle)
    finally:
        lib.pd_plan_destroy(ctx.handle, p)
    return out, list(form), list(mom)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mode", ["vacuum", "weighted"])
def test_globules_sum_directions(gpu_ctx, precision, mode):
    for n, qmax, nq in ((700, 0.3, 60), (3000, 0.5, 200), (9000, 0.8, 120)):
        _, form, mom = _run(gpu_ctx, _request(_globule(n), qmax, nq, precision, mode))
        assert form == [DIRECTIONS] and mom[0] >= 8, (n, form, mom)


def test_extended_structures_sum_pair_moments(gpu_ctx):
    for xyz, qmax, nq in ((_rod(3000, 500.0), 0.5, 300), (_rod(2000, 900.0), 1.0, 600)):
        for mode in ("vacuum", "weighted"):
            _, form, _ = _run(gpu_ctx, _request(xyz, qmax, nq, "fp32", mode))
            assert form[0] in (MOMENTS, GRID if mode == "weighted" else MOMENTS), form


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_every_rank_of_a_shard_sums_directions(gpu_ctx, precision):
    req = _request(_globule(2500), 0.7, 150, precision)
    whole, form, _ = _run(gpu_ctx, req)
    assert form == [DIRECTIONS]
    total = np.zeros_like(whole)
    for rank in range(3):
        out, form, _ = _run(gpu_ctx, req, (rank, 3))
        assert form == [DIRECTIONS], (rank, form)
        total += out
    assert np.all(term_errors(total, whole) < 1e-12)


CASES = ([("fp32", m, 4000, 400) for m in (16, 24, 32, 40, 48, 56)] +
         [("fp32", m, 6000, 400) for m in (64, 72, 80)] +
         [("fp32", m, 12000, 400) for m in (96, 104, 112)] +
         [("fp32", m, 18000, 400) for m in (120, 128)] +
         [("fp32", 136, 20000, 600), ("fp32", 168, 30000, 800)] +
         [("fp64", m, 1500, 400) for m in (24, 32, 40, 48, 56, 64, 72, 128)] +
         [("fp64", m, 3000, 800) for m in (136, 176, 208)])


# The direction kernels are compiled for every 8 (from 64 moments on 16) moments up to
# 128 (FP64: 64), later blocks hold the rest: structures with so many atoms and grid
# points that the directions are the cheaper form at the given moment count.
@pytest.mark.parametrize("precision,moments,n,nq", CASES)
def test_direction_kernels_of_every_moment_count(gpu_ctx, precision, moments, n, nq):
    """The moment count asked for is the one that ran; the last grid point and, for
    small structures, the middle one against the oracle."""
    xyz = _ball(n, 10.0, moments)
    lo, hi = 0.0, 40.0  # the largest q_max whose moments do not exceed the count
    while hi - lo > 0.1:
        q = 0.5 * (lo + hi)
        _, form, mom = _run(gpu_ctx, _request(xyz, q, nq, precision))
        lo, hi = (q, hi) if mom[0] <= moments and form == [DIRECTIONS] else (lo, q)
    req = _request(xyz, lo, nq, precision)
    got, form, mom = _run(gpu_ctx, req)
    assert form == [DIRECTIONS] and mom == [moments], (form, mom)
    qi = np.array([nq // 2, nq - 1] if n < 10000 else [nq - 1])
    err = term_errors(got[:, qi], O.terms_for_request(req, q_index=qi, precise=True))
    assert np.all(err < TOL[precision]), err


def test_cheaper_form_for_few_grid_points(gpu_ctx):
    """A few grid points up to a large q cost less one by one than the directions (or
    pair moments) that the range needs, and more of them do not."""
    for precision in ("fp32", "fp64"):
        for xyz, qmax in ((_ball(4000, 25.0), 4.0), (_rod(3000, 500.0), 0.5)):
            for mode in ("vacuum", "weighted"):
                req = _request(xyz, qmax, 4, precision, mode)
                got, form, _ = _run(gpu_ctx, req)
                assert form == [GRID], (precision, mode, form)
                err = term_errors(got, O.terms_for_request(req, precise=True))
                assert np.all(err < TOL[precision]), err
                _, form, _ = _run(gpu_ctx, _request(xyz, qmax, 600, precision, mode))
                assert form != [GRID] or precision == "fp64", (precision, mode, form)
    # weighted mode: two sums per value make the moments' sequences and flushes weigh more
    _, form, mom = _run(gpu_ctx, _request(_rod(3000, 900.0), 1.0, 500, "fp32", "weighted"))
    assert form == [GRID], (form, mom)


@pytest.mark.parametrize("precision,mode,n,n_species,qmax,nq,want", [
    ("fp64", "weighted", 217, 30, 1.0, 59, GRID), ("fp64", "weighted", 217, 2, 1.0, 59, DIRECTIONS),
    ("fp64", "vacuum", 1000, 60, 1.0, 60, GRID), ("fp64", "vacuum", 1000, 4, 1.0, 60, DIRECTIONS),
    ("fp64", "weighted", 300, 16, 2.0, 300, GRID), ("fp64", "vacuum", 300, 1, 2.0, 300, DIRECTIONS),
    ("fp32", "weighted", 500, 30, 0.5, 12, GRID), ("fp32", "weighted", 500, 2, 0.5, 12, DIRECTIONS),
    ("fp32", "vacuum", 10000, 60, 1.0, 60, MOMENTS), ("fp32", "vacuum", 10000, 2, 1.0, 60, DIRECTIONS),
    ("fp32", "vacuum", 2000, 84, 1.0, 1000, DIRECTIONS)])
def test_many_classes_and_the_form(gpu_ctx, precision, mode, n, n_species, qmax, nq, want):
    """The directions form every class pair's products at every node, the tiles of small
    classes are short: the form follows the class count, and a solve, which decides on the
    host, agrees with a plan's execution."""
    rng = np.random.default_rng(n + n_species)
    sp = rng.integers(0, n_species, n)
    ff = rng.uniform(1, 8, (n_species, nq))
    xyz = _ball(n, 1.6 * n ** (1 / 3))
    extra = ((None,) * 3 if mode == "vacuum" else
             (rng.uniform(0.2, 3, (n_species, nq)), rng.uniform(0, 2, n), rng.uniform(5, 10, nq)))
    req = DebyeRequest(xyz, sp, ff, *extra, 0.0, qmax, nq, None, precision)
    got, form, _ = _run(gpu_ctx, req)
    assert form == [want] or (want != DIRECTIONS and form != [DIRECTIONS]), form
    qi = np.array([0, nq // 2, nq - 1])
    err = term_errors(got[:, qi], O.terms_for_request(req, q_index=qi, precise=True))
    assert np.all(err < TOL[precision]), err
    both = term_errors(solve(req, gpu_ctx), got)
    assert np.all(both < (1e-13 if precision == "fp64" else 1e-6)), both


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_frames_of_a_batch_take_their_own_form(gpu_ctx, precision):
    xyz = _globule(800)
    far = 8.0 if precision == "fp32" else 15.0  # (a grid point costs a double sin)
    frames = np.stack([xyz, far * xyz, xyz + 1.0])
    _, form, _ = _run(gpu_ctx, _request(frames, 0.6, 45, precision))
    assert form[0] == form[2] == DIRECTIONS and form[1] != DIRECTIONS, form


@pytest.mark.parametrize("precision,n,n_frames", [
    ("fp64", 9, 1), ("fp64", 9, 148), ("fp64", 9, 149), ("fp64", 9, 296), ("fp64", 9, 297),
    ("fp64", 9, 700), ("fp64", 150, 3), ("fp32", 40, 148), ("fp32", 40, 445), ("fp32", 40, 900)])
def test_every_job_is_taken_once(gpu_ctx, precision, n, n_frames):
    """Fewer jobs than blocks, as many, and more: a block's first job is its own number and
    the others are drawn. Each frame has its own weight, so a job left out or taken twice
    shows; the frames' mean against the compensated oracle."""
    rng = np.random.default_rng(n_frames)
    frames = rng.uniform(-9, 9, (n_frames, n, 3))
    req = _request(frames, 0.6, 20, precision)
    req.frame_weights = rng.uniform(0.1, 2.0, n_frames)
    want = 0.0
    for x, w in zip(frames, req.frame_weights):
        one = DebyeRequest(x, req.species, req.ff_atoms, None, None, None, 0.0, 0.6, 20, None,
                           precision)
        want = want + w * O.terms_for_request(one, q_index=np.array([0, 7, 19]), precise=True)
    err = term_errors(solve(req, gpu_ctx)[:, [0, 7, 19]], want / req.frame_weights.sum())
    assert np.all(err < TOL[precision]), err
