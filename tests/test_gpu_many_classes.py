"""Requests with more species than the atom classes of the (species, weight) split:
a class per species, without a bound.

pd_profiles stages the class factors in shared memory up to about 85 classes
(512 moments) and reads them from L2 beyond; the class counts lie on both sides
of that line. Tolerances are those of the two forms: FP64 1e-10 and FP32 1e-5 of
the compensated oracle."""
import numpy as np
import pytest

from conftest import term_errors
from oracle import oracle as O
from pripps_b200.debye import DebyeRequest, TrajectoryStream, solve

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-10, "fp32": 1e-5}


def _request(n, n_species, nq, precision, mode, seed):
    rng = np.random.default_rng(seed)
    sp = np.concatenate([np.arange(n_species), rng.integers(0, n_species, n - n_species)])
    rng.shuffle(sp)
    ff = rng.uniform(1, 8, (n_species, nq))
    xyz = rng.uniform(-14, 14, (n, 3))
    if mode == "vacuum":
        return DebyeRequest(xyz, sp, ff, None, None, None, 0.0, 0.6, nq, None, precision)
    return DebyeRequest(xyz, sp, ff, rng.uniform(0.2, 3, (n_species, nq)), rng.uniform(0, 2, n),
                        rng.uniform(5, 10, nq), 0.0, 0.6, nq, None, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mode,n,n_species,nq", [("vacuum", 900, 85, 520), ("vacuum", 900, 86, 520),
                                                 ("vacuum", 900, 100, 520),
                                                 ("weighted", 700, 100, 520),
                                                 ("vacuum", 900, 400, 600),
                                                 ("weighted", 450, 300, 500),
                                                 ("vacuum", 1600, 1500, 500),
                                                 ("vacuum", 300, 230, 3)])
def test_species_without_a_bound(gpu_ctx, precision, mode, n, n_species, nq):
    req = _request(n, n_species, nq, precision, mode, n_species)
    qi = np.unique([0, 1, nq // 2, nq - 1])
    got = solve(req, gpu_ctx)
    err = term_errors(got[:, qi], O.terms_for_request(req, q_index=qi, precise=True))
    assert np.all(err < TOL[precision]), err


@pytest.mark.parametrize("mode,n_species,nq,n_frames", [
    ("vacuum", 30, 1184, 1), ("vacuum", 30, 1185, 1), ("vacuum", 30, 400, 9),
    ("vacuum", 5, 60, 1), ("weighted", 30, 1184, 1), ("weighted", 30, 1185, 1),
    ("weighted", 30, 60, 60), ("weighted", 100, 30, 1), ("vacuum", 250, 30, 1)])
def test_steps_of_staged_pair_rows(gpu_ctx, mode, n_species, nq, n_frames):
    """Moments of the pairs of an elongated set: both sides of the block counts where the
    steps change their length, one step and many, whole and with a last short one; every
    profile against the compensated oracle, frames as the weighted mean."""
    rng = np.random.default_rng(n_species * nq)
    req = _request(140 if n_species < 100 else 300, n_species, nq, "fp32", mode, nq)
    req.xyz = req.xyz * np.array([6.0, 0.5, 0.5])
    qi = np.unique([0, 1, nq // 2, nq - 1])
    if n_frames == 1:
        got = solve(req, gpu_ctx)
        err = term_errors(got[:, qi], O.terms_for_request(req, q_index=qi, precise=True))
        assert np.all(err < TOL["fp32"]), err
        return
    base, frames = req.xyz, []
    weights = rng.uniform(0.1, 2, n_frames)
    want = 0.0
    for k in range(n_frames):
        req.xyz = base * rng.uniform(0.6, 1.0) + rng.normal(0, 0.3, base.shape)
        frames.append(req.xyz)
        want = want + weights[k] * O.terms_for_request(req, q_index=qi, precise=True)
    req.xyz, req.frame_weights = np.stack(frames), weights
    got = solve(req, gpu_ctx)
    err = term_errors(got[:, qi], want / weights.sum())
    assert np.all(err < TOL["fp32"]), err


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_many_species_in_a_stream(gpu_ctx, precision):
    """The same through a streamed trajectory: the mean of the frames' own solves."""
    req = _request(400, 120, 500, precision, "vacuum", 3)
    frames = req.xyz[None] + np.random.default_rng(4).normal(0, 0.3, (3, 400, 3))
    s = TrajectoryStream(req, 2, gpu_ctx)
    s.push(frames, None)
    want = []
    for x in frames:
        req.xyz = x
        want.append(solve(req, gpu_ctx))
    tol = 1e-12 if precision == "fp64" else 1e-5
    assert np.all(term_errors(s.finish(), np.mean(want, axis=0)) < tol)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_excluded_dummies_with_a_weight_each(gpu_ctx, precision):
    """A caller's excluded-volume set with 300 distinct weights (one species each in
    the joint request) against the reference's sets."""
    from pripps_b200.debye import union_request
    from pripps_b200.dummies import DummySet
    from pripps_b200.formfactor import SingleGaussian, linear_q_values
    rng = np.random.default_rng(11)
    n, m, nq = 250, 330, 500
    q = linear_q_values(0.0, 0.5, nq)
    pos = rng.uniform(-12, 12, (n, 3))
    sp = rng.integers(0, 3, n)
    ffa = rng.uniform(1, 8, (3, nq))
    w = np.concatenate([np.linspace(5.0, 40.0, 300), rng.choice(np.linspace(5.0, 40.0, 300), m - 300)])
    exc = DummySet.weighted(rng.uniform(-12, 12, (m, 3)), SingleGaussian(1.0, 1.5), w)
    req = union_request(pos, sp, ffa, None, None, None, exc, None, q, 0.0, 0.5, precision)
    qi = np.array([0, 1, 250, 499])
    got = solve(req, gpu_ctx)
    idx, rows = exc.rows(q)
    assert len(rows) == 300
    ref = O.build_model_sets(pos, sp, ffa, exc.positions, idx, rows, qmin=0.0, qmax=0.5, nq=nq,
                             q_index=qi).T
    err = term_errors(got[:, qi], ref)
    assert np.all(err < TOL[precision]), err
