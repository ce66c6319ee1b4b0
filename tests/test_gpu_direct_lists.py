"""Which lattice vectors go to the line kernel, and what looking for lines costs."""
import time

import numpy as np
import pytest

from pripps_b200 import _lib
from pripps_b200.direct import amplitudes, miller_indices

pytestmark = pytest.mark.gpu
BOX = np.array([60.0, 61.0, 62.0])


def _lists():
    rng = np.random.default_rng(2)
    half = np.array([(h, k, l) for h in range(13) for k in range(-12, 13) for l in range(-12, 13)
                     if h * h + k * k + l * l <= 144])
    yield "miller", miller_indices(60), True
    yield "miller_shuffled", rng.permutation(miller_indices(60)), True
    yield "filled", half, True
    yield "filled_shuffled", rng.permutation(half), True
    yield "along_k", np.array([(h, k, l) for h in (-3, 500) for l in (-512, 7)
                               for k in range(-512, -400)]), True
    yield "two_thousand_and_more", np.array([(h, k, l) for h in range(13) for k in range(13)
                                             for l in range(-512, 513, 1)])[::1][:30000], True
    yield "every_third", half[rng.random(len(half)) < 0.33], False
    yield "scattered", rng.integers(-512, 513, (5000, 3)), False
    yield "scattered_small", rng.integers(-40, 41, (3000, 3)), False
    yield "one", np.array([[0, 0, 0]]), False


@pytest.mark.parametrize("name,hkl,lines", list(_lists()), ids=lambda v: v if type(v) is str else "")
def test_lists_and_their_kernels(gpu_ctx, name, hkl, lines):
    """Lists on lines take three kernels (sort, lines, reduction), others two; both
    give pd_direct's rows. 1e-12 of Σ|f|, the tolerance of the entry points."""
    rng = np.random.default_rng(len(hkl))
    n, nk = 260, 3
    xyz, kind = rng.uniform(-60, 60, (n, 3)), rng.integers(0, nk, n)
    ff = rng.uniform(-2, 8, (nk, len(hkl)))
    before = _lib.lib().pd_launch_count(gpu_ctx.handle)
    got = amplitudes(xyz, kind, ff, None, 2, None, gpu_ctx, hkl=hkl, box=BOX)
    assert _lib.lib().pd_launch_count(gpu_ctx.handle) - before == (3 if lines else 2)
    ref = amplitudes(xyz, kind, ff, 2 * np.pi * hkl / BOX, 2, None, gpu_ctx)
    scale = np.sum(np.abs(ff[kind]), axis=0)
    assert np.all(np.abs(got[:, :2] - ref[:, :2]) <= 1e-12 * scale[:, None])
    assert np.all(np.abs(got[:, 2:] - ref[:, 2:]) <= 2e-12 * scale[:, None] ** 2)


def test_scattered_vectors_cost_no_search(gpu_ctx):
    """100,000 scattered vectors: a call that looks for lines (molecules of 200 points)
    against one that does not (100 points): the search is a small part of it. (It
    sorted the list by every kind of line first: eight times the call.)"""
    rng = np.random.default_rng(4)
    hkl = rng.integers(-60, 61, (100_000, 3))
    n = 400
    xyz, kind = rng.uniform(-60, 60, (n, 3)), rng.integers(0, 2, n)
    ff = rng.uniform(1, 8, (2, len(hkl)))

    def best(n_mol):
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            amplitudes(xyz, kind, ff, None, n_mol, None, gpu_ctx, hkl=hkl, box=BOX)
            t.append(time.perf_counter() - t0)
        return min(t)
    assert best(2) < 1.5 * best(4)


@pytest.mark.parametrize("n_mol,mol,nk", [(1, 4095, 3), (1, 4096, 2), (1, 4097, 4), (2, 9001, 5),
                                          (1, 30000, 32), (3, 128, 1)])
def test_molecules_sorted_in_pieces(gpu_ctx, n_mol, mol, nk):
    """The points are grouped by kind in pieces of 4,096 and the line kernel's slices
    cut across them: every point counts once, with its own weight."""
    rng = np.random.default_rng(mol)
    n, hkl = n_mol * mol, miller_indices(20)
    xyz, kind, w = rng.uniform(-60, 60, (n, 3)), rng.integers(0, nk, n), rng.uniform(0, 2, n)
    ff = rng.uniform(-2, 8, (nk, len(hkl)))
    for weight in (None, w):
        before = _lib.lib().pd_launch_count(gpu_ctx.handle)
        got = amplitudes(xyz, kind, ff, None, n_mol, weight, gpu_ctx, hkl=hkl, box=BOX)
        assert _lib.lib().pd_launch_count(gpu_ctx.handle) - before == 3
        ref = amplitudes(xyz, kind, ff, 2 * np.pi * hkl / BOX, n_mol, weight, gpu_ctx)
        scale = np.sum(np.abs(ff[kind]) * (1.0 if weight is None else w[:, None]), axis=0)
        assert np.all(np.abs(got[:, :2] - ref[:, :2]) <= 1e-12 * scale[:, None])
        assert np.all(np.abs(got[:, 2:] - ref[:, 2:]) <= 2e-12 * scale[:, None] ** 2)


def test_one_large_molecule_is_no_slower_than_many(gpu_ctx):
    """A million points as one molecule against 64 molecules: the same points and vectors,
    and the points of one molecule are not left to one SM."""
    rng = np.random.default_rng(6)
    hkl, n = miller_indices(100), 1_000_000
    xyz, kind = rng.uniform(-60, 60, (n, 3)), rng.integers(0, 3, n)
    ff = rng.uniform(1, 8, (3, len(hkl)))

    def best(n_mol):
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            amplitudes(xyz, kind, ff, None, n_mol, None, gpu_ctx, hkl=hkl, box=BOX)
            t.append(time.perf_counter() - t0)
        return min(t)
    assert best(1) < 1.25 * best(64)
