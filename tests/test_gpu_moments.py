"""The moment form of the pair sum at the sizes where it can go wrong.

Every pair's sinc(q r) is expanded in cos(n φ), sin(φ/2) = r/d; the number of
moments grows with q_max·d, they are summed in blocks of the kernel shape's
size, and the q-block jobs of a tile become parts of its j range. The cases
put the moment count below, at and above a block for every block size, leave
jobs idle (more q-blocks than blocks × parts use), and reach the bounds of the
rule (few grid points on a long range: the grid points are summed directly).

Tolerances are those of the two forms: FP64 1e-10 and FP32 1e-5 of the
compensated oracle, self profiles relative and cross profiles normalised (an
FP32 moment carries rounding errors of at most n·6e-8 per pair with random
signs, n <= 512; the worst single pair, two atoms at the largest distance, is
below 512·6e-8/(z/2) <= 4e-7 of its value's scale).
"""
import numpy as np
import pytest

from conftest import term_errors
from oracle import oracle as O
from pripps_b200 import _lib, workloads
from pripps_b200.debye import DebyeRequest, TrajectoryStream, solve

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-10, "fp32": 1e-5}


def _request(xyz, nq, qmin, qmax, precision, mode, seed):
    rng = np.random.default_rng(seed)
    n = len(xyz)
    sp = rng.integers(0, 3, n)
    ff = rng.uniform(1, 8, (3, nq))
    if mode == "vacuum":
        return DebyeRequest(xyz, sp, ff, None, None, None, qmin, qmax, nq, None, precision)
    w = rng.uniform(0, 2, n) if mode == "weighted" else np.where(rng.random(n) < 0.5, 1.25, 0.0)
    return DebyeRequest(xyz, sp, ff, rng.uniform(0.2, 3, (3, nq)), w, rng.uniform(5, 10, nq),
                        qmin, qmax, nq, None, precision)


def _check(req, ctx, precision):
    t = solve(req, ctx)
    qi = np.unique(np.concatenate([np.arange(min(4, req.nq)), [req.nq // 2],
                                   np.arange(max(0, req.nq - 2), req.nq)]))
    ref = O.terms_for_request(req, q_index=qi, precise=True)
    err = term_errors(t[:, qi], ref)
    assert np.all(err < TOL[precision]), err


# radius × qmax sets z = q_max·d ≈ 2.06·radius·qmax, so about z/2 + 5·z^(1/3) moments:
# 8, 24, 32/33 (a block of 32), 64, 128 (one block of 128), 145 (two), 300 and
# 500 (several; with nq = 90 more than the rule allows)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mode", ["vacuum", "class", "weighted"])
@pytest.mark.parametrize("radius,qmax,nq", [(1.0, 0.3, 40), (16.0, 0.5, 61), (18.0, 0.98, 100),
                                            (18.0, 1.02, 100), (40.0, 1.02, 257), (60.0, 1.5, 300),
                                            (60.0, 2.1, 129), (90.0, 2.9, 400), (150.0, 3.0, 600),
                                            (150.0, 3.0, 90)])
def test_moment_counts(gpu_ctx, precision, mode, radius, qmax, nq):
    rng = np.random.default_rng(int(radius * 100 + nq))
    n = 333
    v = rng.normal(size=(n, 3))
    xyz = radius * v / np.linalg.norm(v, axis=1)[:, None] * rng.random((n, 1)) ** (1 / 3)
    _check(_request(xyz, nq, 0.02 if nq == 61 else 0.0, qmax, precision, mode, nq), gpu_ctx,
           precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(32, 4), (64, 2), (64, 4), (96, 2), (128, 1), (128, 4),
                                   (160, 1), (192, 1)])
@pytest.mark.parametrize("tj", [32, 96, 512])
def test_moment_blocks_of_every_shape(precision, shape, tj):
    """Moment block and slot stride differ between the shapes, and a part of a
    short j range may be empty."""
    K, NP = shape
    if precision == "fp64":
        K, NP = (16 if K == 32 else 32), 1
    ctx = _lib.Context(0)
    try:
        rng = np.random.default_rng(K + tj)
        n, nq = 700, 290
        _lib.check(_lib.lib().pd_set_tuning(ctx.handle, n, nq, _lib.PRECISIONS[precision], K, tj,
                                            NP), ctx.handle)
        xyz = rng.uniform(-20, 20, (n, 3))
        _check(_request(xyz, nq, 0.0, 1.2, precision, "class", K), ctx, precision)
    finally:
        ctx.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("name", ["one", "pair", "coincident", "all_coincident", "line", "far"])
def test_moment_extreme_distances(gpu_ctx, precision, name):
    """Distances at the ends of the expansion: r = 0 (also with a zero radius),
    and r = 2·radius, the largest φ."""
    rng = np.random.default_rng(5)
    xyz = {"one": np.zeros((1, 3)),
           "pair": np.array([[0, 0, 0], [37.0, 0, 0]]),
           "coincident": np.array([[1, 2, 3], [1, 2, 3], [9.0, -2, 4]]),
           "all_coincident": np.full((40, 3), 2.5),
           "line": np.stack([np.linspace(-60, 60, 131), np.zeros(131), np.zeros(131)], axis=1),
           "far": np.concatenate([rng.normal(size=(60, 3)), rng.normal(size=(60, 3)) + 150.0])}
    _check(_request(xyz[name], 200, 0.0, 0.8, precision, "vacuum", 3), gpu_ctx, precision)


# The direction form (amplitudes over a quadrature of the sphere) runs where
# there are more atoms than directions: sizes around the chunk length (1,024), a
# chunk of one atom, several chunks of a class; z = 2·radius·qmax of a few rings,
# of 33/64/65 directions' worth of moments, and past one moment block; 49 grid
# points that hit an interpolation node (qmin = qmax·cos(π/4M) is not on the grid:
# q = 0 and the ends are the exact cases).
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mode", ["vacuum", "class", "weighted"])
@pytest.mark.parametrize("n,qmax,nq,qmin", [(700, 0.15, 30, 0.0), (1025, 0.4, 49, 0.02),
                                            (1536, 0.5, 65, 0.5), (1300, 1.2, 129, 0.0),
                                            (2100, 2.3, 140, 0.0)])
def test_direction_form(gpu_ctx, precision, mode, n, qmax, nq, qmin):
    from pripps_b200 import synth
    rng = np.random.default_rng(n)
    r = synth.sphere_radius_for(n)
    xyz = synth.rsa_points(n, (r, r, r), rng)
    req = _request(xyz, nq, qmin, qmax, precision, mode, n)
    req.species[:] = rng.choice(3, size=n, p=[0.6, 0.4 - 1.0 / n, 1.0 / n])
    _check(req, gpu_ctx, precision)


# A direction unit is compiled for every 8 (from 64 moments on 16) moments up to
# 128 (FP64: 64), later blocks hold the rest: each of them, with the two grid points
# that leave large moment counts to this form (a grid point direct: 1,500 atoms'
# pairs); radius and order as in the form's own rule.
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mode", ["vacuum", "weighted"])
@pytest.mark.parametrize("moments", [8, 16, 24, 32, 40, 48, 56, 64, 72, 80, 96, 104, 112, 120, 128,
                                     136, 168, 240])
def test_direction_moment_counts(gpu_ctx, precision, mode, moments):
    a, b = (13.0, 3.0) if precision == "fp64" else (8.0, 2.0)
    z = np.linspace(0.0, 300.0, 30001)
    z = z[np.searchsorted(z + a * np.cbrt(0.5 * z) + b, max(moments - 4.0, b + 0.1))]
    rng = np.random.default_rng(moments)
    v = rng.normal(size=(1500, 3))
    xyz = v / np.linalg.norm(v, axis=1)[:, None] * rng.random((1500, 1)) ** (1 / 3)
    xyz -= xyz.mean(axis=0)
    xyz *= 10.0 / np.linalg.norm(xyz, axis=1).max()
    _check(_request(xyz, 2, 0.0, z / 10.3, precision, mode, moments), gpu_ctx, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_direction_form_shards_add_up(precision):
    """Ranks take whole groups of directions; three ranks' partial profiles (run
    one after another) add up to the whole solve."""
    import ctypes as C

    import torch
    lib = _lib.lib()
    ctx = _lib.Context(0)
    try:
        rng = np.random.default_rng(8)
        xyz = rng.uniform(-22, 22, (2500, 3))
        req = _request(xyz, 150, 0.0, 0.7, precision, "class", 8)
        r = req.c_struct()
        whole = solve(req, ctx)
        dev = torch.from_numpy(req.xyz).cuda()
        total = np.zeros((6, req.nq))
        for rank in range(3):
            p = C.c_void_p()
            _lib.check(lib.pd_plan_create(ctx.handle, C.byref(r), C.byref(p)), ctx.handle)
            _lib.check(lib.pd_plan_set_shard(ctx.handle, p, rank, 3), ctx.handle)
            out = torch.empty((6, req.nq), dtype=torch.float64, device="cuda")
            _lib.check(lib.pd_plan_execute(ctx.handle, p, dev.data_ptr(), out.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream), ctx.handle)
            torch.cuda.synchronize()
            total += out.cpu().numpy()
            lib.pd_plan_destroy(ctx.handle, p)
        assert np.all(term_errors(total, whole) < 1e-12)
    finally:
        ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_frames_of_both_forms_share_a_batch(gpu_ctx, precision):
    """A batch whose frames take different forms (a globule sums directions, the
    same points blown up eight times need more directions than there are pairs):
    every frame keeps its own sums. The frames of the batch are solved one by
    one for comparison; FP64 rounding, and the FP32 sums' grouping."""
    w = workloads.small_globule(800, 5, nq=45, solvent=False, precision=precision)
    rng = np.random.default_rng(8)
    frames = w.request.xyz[None] + rng.normal(0, 0.4, (12, 800, 3))
    frames[::3] *= 8.0
    weights = rng.exponential(1.0, 12)
    r = w.request

    def req(xyz, fw):
        return DebyeRequest(xyz, r.species, r.ff_atoms, None, None, None, r.qmin, r.qmax, r.nq,
                            fw, precision)
    want = sum(f * solve(req(x, None), gpu_ctx) for f, x in zip(weights, frames)) / weights.sum()
    s = TrajectoryStream(req(r.xyz, None), 12, gpu_ctx)
    s.push(frames, weights)
    tol = 1e-12 if precision == "fp64" else 1e-5
    assert np.all(term_errors(s.finish(), want) < tol)
    assert np.all(term_errors(solve(req(frames, weights), gpu_ctx), want) < tol)


@pytest.mark.parametrize("n", [120, 900, 17000])
def test_plan_execution_replays_from_a_graph(gpu_ctx, n):
    """A plan's chained kernels (pairs; directions; the separate centroid and pack
    kernels above 16,384 atoms) captured into a CUDA graph: every replay gives the
    direct execution's result for the coordinates of that moment, bit for bit."""
    import torch

    from pripps_b200.shard import ShardedPlan
    w = workloads.small_globule(min(n, 2000), 6, nq=50, precision="fp32").request
    if n > 2000:
        rng = np.random.default_rng(n)
        xyz = rng.uniform(-25.0, 25.0, (n, 3))
        w = _request(xyz, 50, 0.0, 0.3, "fp32", "vacuum", n)
    plan = ShardedPlan(w, gpu_ctx, 0, 1)
    try:
        xyz = torch.tensor(w.xyz, device="cuda")
        want = plan.execute(xyz).clone()
        moved = xyz * 1.03
        want2 = plan.execute(moved).clone()
        buf, s = xyz.clone(), torch.cuda.Stream()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            out = plan.execute(buf)
        for src, ref in ((xyz, want), (moved, want2), (xyz, want)):
            buf.copy_(src)
            g.replay()
            torch.cuda.synchronize()
            assert torch.equal(out, ref)
    finally:
        plan.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_coincident_points_at_large_q(gpu_ctx, precision):
    """A radius of zero: the expansion's own radius is bounded from below, on the
    host that sizes the tables as on the device that fills them."""
    xyz = np.full((300, 3), 1.5)
    _check(_request(xyz, 4, 0.0, 5e4, precision, "vacuum", 2), gpu_ctx, precision)
