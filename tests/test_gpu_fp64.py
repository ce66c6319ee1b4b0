"""The FP64 form keeps double precision in every profile point, deep minima included.

A point is a sum of N² terms of both signs, 1e-2 to 1e-5 of what it is at q = 0
here. Tolerance 5e-15 of a point against sums in long double (the oracle's cross
profiles, whose terms are products of doubles, are themselves 1e-14 off): a pair's
term is rounded to 2e-16 with random signs, a thread's run of up to 4,096 of them to
about ten times that; twice their sum is allowed. (Sums over moments of the pairs of
size N², or an interpolation between points of very different size, lose a digit or
more.) Directions: 1e-14; an amplitude is a sum over N atoms, rounded to 1e-16·√N and
a few times that, of the size of √N where the profile is deep; that share of it
averages over the directions, and the rule's weights and the Bessel coefficients add
1e-15; a factor of three is to spare.
"""
import numpy as np
import pytest

from conftest import term_errors
from pripps_b200.debye import DebyeRequest, solve

pytestmark = pytest.mark.gpu
TOL, TOL_DIRECTIONS = 5e-15, 1e-14


def _long_double(req, qi):
    """The six profiles at grid points qi, every operation in long double."""
    x = req.xyz.astype(np.longdouble)
    i, j = np.triu_indices(len(x), 1)
    r = np.sqrt(((x[i] - x[j]) ** 2).sum(axis=1))
    w = np.zeros(len(x)) if req.hyd_weights is None else req.hyd_weights
    out = np.zeros((6, len(qi)))
    for k, q in enumerate(qi):
        z = r * np.longdouble(req.qmin + (req.qmax - req.qmin) * q / (req.nq - 1))
        s = np.sin(z) / np.where(z > 0, z, 1) if q else np.ones_like(z)
        f = [req.ff_atoms[req.species, q].astype(np.longdouble)]
        f.append(0 * f[0] if req.ff_excluded is None else
                 req.ff_excluded[req.species, q].astype(np.longdouble))
        f.append(0 * f[0] if req.ff_water is None else w * np.longdouble(req.ff_water[q]))
        for row, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            u, v = f[a], f[b]
            out[row, k] = ((u[i] * v[j] + u[j] * v[i]) * s).sum() + (u * v).sum()
    return out


def _check(xyz, qmax, nq, mode, ctx, tol=TOL):
    rng = np.random.default_rng(len(xyz))
    n = len(xyz)
    sp = rng.integers(0, 3, n)
    ff = rng.uniform(1, 8, (3, nq))
    if mode == "vacuum":
        req = DebyeRequest(xyz, sp, ff, None, None, None, 0.0, qmax, nq, None, "fp64")
    else:
        w = rng.uniform(0, 2, n) if mode == "weighted" else np.where(rng.random(n) < 0.5, 1.25, 0.0)
        req = DebyeRequest(xyz, sp, ff, rng.uniform(0.2, 3, (3, nq)), w, rng.uniform(5, 10, nq),
                           0.0, qmax, nq, None, "fp64")
    got = solve(req, ctx)
    qi = np.unique(np.linspace(0, nq - 1, 10).astype(int))
    err = term_errors(got[:, qi], _long_double(req, qi))
    assert np.all(err < tol), err


def _rod(n, length):
    rng = np.random.default_rng(1)
    xy = rng.uniform(-1, 1, (4 * n, 2))
    xy = xy[(xy ** 2).sum(axis=1) < 1][:n] * 10.0
    return np.column_stack([xy, rng.uniform(-length / 2, length / 2, n)])


@pytest.mark.parametrize("mode", ["vacuum", "class", "weighted"])
@pytest.mark.parametrize("n,length,qmax,nq", [(1500, 400.0, 0.5, 150), (1200, 900.0, 1.0, 300),
                                              (100, 60.0, 0.8, 200)])
def test_pairs(gpu_ctx, mode, n, length, qmax, nq):
    _check(_rod(n, length), qmax, nq, mode, gpu_ctx)


@pytest.mark.parametrize("mode", ["vacuum", "class", "weighted"])
@pytest.mark.parametrize("n,radius,ratio,qmax,nq", [(12, 4.0, 1.0, 0.5, 17), (60, 7.0, 1.0, 1.0, 100),
                                                    (700, 14.0, 1.0, 0.5, 97),
                                                    (1500, 18.0, 1.0, 0.6, 200),
                                                    (1200, 17.0, 2.5, 1.0, 64),
                                                    (1400, 12.0, 1.0, 4.0, 80)])
def test_directions(gpu_ctx, mode, n, radius, ratio, qmax, nq):
    """Balls and an ellipsoid of uniform density: their profiles have minima of 1e-3 to
    1e-4 of the value at q = 0 (the last: several moment blocks)."""
    rng = np.random.default_rng(n)
    v = rng.normal(size=(n, 3))
    xyz = radius * v / np.linalg.norm(v, axis=1)[:, None] * rng.random((n, 1)) ** (1 / 3)
    _check(xyz * np.array([ratio, ratio ** -0.5, ratio ** -0.5]), qmax, nq, mode, gpu_ctx,
           TOL_DIRECTIONS)
