"""Extended structures: rods and chains whose quadrature would need more directions
than they have pairs, so that the pairs' moments are summed.

The close pairs of a long structure have small angles φ (sin(φ/2) = r/d); an error of
their phases with one sign for all of them shows in every profile point. The FP32
form is compared with the FP64 form point by point, all six profiles. Tolerance
2e-6: the FP32 positions alone (6e-8 of half the length, random signs) give up to 3e-7
of a point on such rods with unit weights, the moments are sums over 128 pairs of
FP32 terms, whose rounding is random and of the same size; the profiles of half of
the atoms double that, and a factor of two is to spare.
The FP64 form against the compensated oracle: 1e-12 (2e9 finer rounding; its
expansion is cut at 1e-15 of a pair's term, and a profile point is at least 1e-3
of the sum of the terms here).
"""
import numpy as np
import pytest

from conftest import term_errors
from oracle import oracle as O
from pripps_b200 import _lib
from pripps_b200.debye import DebyeRequest, solve

pytestmark = pytest.mark.gpu


def _rod(n, length, rng, radius=10.0):
    xy = rng.uniform(-1, 1, (4 * n, 2))
    xy = xy[(xy ** 2).sum(axis=1) < 1][:n] * radius
    return np.column_stack([xy, rng.uniform(-length / 2, length / 2, n)])


def _chain(n, rng):
    v = rng.normal(size=(n, 3))
    for i in range(1, n):  # a persistence of about ten steps
        v[i] = 0.9 * v[i - 1] + np.sqrt(1 - 0.81) * v[i]
    return np.cumsum(1.5 * v / np.linalg.norm(v, axis=1)[:, None], axis=0)


def _request(xyz, qmax, nq, precision, mode, seed):
    rng = np.random.default_rng(seed)
    n = len(xyz)
    sp = rng.integers(0, 3, n)
    ff = rng.uniform(1, 8, (3, nq))
    w = rng.uniform(0, 2, n) if mode == "weighted" else np.where(rng.random(n) < 0.5, 1.25, 0.0)
    return DebyeRequest(xyz, sp, ff, rng.uniform(0.2, 3, (3, nq)), w, rng.uniform(5, 10, nq),
                        0.0, qmax, nq, None, precision)


def _structure(name, rng):
    return {"rod500": lambda: (_rod(5000, 500.0, rng), 0.5, 300),
            "rod900": lambda: (_rod(6000, 900.0, rng), 1.0, 500),
            "chain": lambda: (_chain(10000, rng), 1.0, 400)}[name]()


# moment blocks of 128 (one, and several of them), 64 and 32; the weighted mode in
# its own shape
@pytest.mark.parametrize("name", ["rod500", "rod900", "chain"])
@pytest.mark.parametrize("mode,K,NP", [("class", 128, 4), ("class", 64, 4), ("class", 32, 4),
                                       ("weighted", 0, 0)])
def test_extended_structures_fp32(name, mode, K, NP):
    xyz, qmax, nq = _structure(name, np.random.default_rng(3))
    ctx = _lib.Context(0)
    try:
        if K:
            _lib.check(_lib.lib().pd_set_tuning(ctx.handle, len(xyz), nq, 0, K, 512, NP),
                       ctx.handle)
        got = solve(_request(xyz, qmax, nq, "fp32", mode, 1), ctx)
        want = solve(_request(xyz, qmax, nq, "fp64", mode, 1), ctx)
    finally:
        ctx.close()
    err = term_errors(got, want)
    assert np.all(err < 2e-6), err


@pytest.mark.parametrize("name", ["rod500", "rod900"])
@pytest.mark.parametrize("mode", ["class", "weighted"])
def test_extended_structures_fp64(gpu_ctx, name, mode):
    xyz, qmax, nq = _structure(name, np.random.default_rng(3))
    req = _request(xyz, qmax, nq, "fp64", mode, 1)
    qi = np.array([1, nq // 3, 2 * nq // 3, nq - 1])
    err = term_errors(solve(req, gpu_ctx)[:, qi], O.terms_for_request(req, q_index=qi,
                                                                     precise=True))
    assert np.all(err < 1e-12), err
