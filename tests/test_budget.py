"""Device memory of a request in its smallest layout (host-only): what a context's
budget, or the fixed scratch of pd_solve_noalloc, refuses it by. The layouts of the
moment and direction forms must not refuse what ran with the grid points alone; the
ceilings are the bytes those took."""
import ctypes as C

import numpy as np
import pytest

from pripps_b200 import _lib
from pripps_b200.debye import DebyeRequest

# n, nq, species, precision, mode, frames, bytes
CASES = [(100, 24, 1, 'fp64', 'vacuum', 1, 13568),
         (300, 100, 4, 'fp64', 'vacuum', 1, 58368),
         (1700, 1300, 3, 'fp64', 'class', 1, 1627648),
         (540, 20, 1, 'fp64', 'weighted', 1, 45312),
         (1500, 82, 5, 'fp32', 'class', 1, 224256),
         (3000, 300, 4, 'fp32', 'class', 1, 942080),
         (20000, 512, 4, 'fp32', 'weighted', 1, 17490944),
         (2000, 700, 5, 'fp32', 'weighted', 1, 3126272),
         (500, 68, 7, 'fp32', 'weighted', 16, 3793152),
         (5000, 300, 4, 'fp32', 'vacuum', 64, 29802496),
         (900, 12, 90, 'fp32', 'vacuum', 1, 1816576),
         (1200, 300, 200, 'fp32', 'vacuum', 1, 103313664),
         (100000, 1000, 4, 'fp32', 'class', 1, 34851840)]


def _request(n, nq, n_species, precision, mode, frames):
    rng = np.random.default_rng(n + nq)
    xyz = rng.uniform(-20, 20, (frames, n, 3) if frames > 1 else (n, 3))
    sp = rng.integers(0, n_species, n)
    ff = rng.uniform(1, 8, (n_species, nq))
    if mode == "vacuum":
        return DebyeRequest(xyz, sp, ff, None, None, None, 0.0, 0.5, nq, None, precision)
    w = rng.uniform(0, 2, n) if mode == "weighted" else np.where(rng.random(n) < 0.3, 1.25, 0.0)
    return DebyeRequest(xyz, sp, ff, ff, w, ff[0], 0.0, 0.5, nq, None, precision)


@pytest.mark.parametrize("n,nq,n_species,precision,mode,frames,ceiling", CASES)
def test_smallest_layout_has_not_grown(n, nq, n_species, precision, mode, frames, ceiling):
    req = _request(n, nq, n_species, precision, mode, frames)
    r, got = req.c_struct(), C.c_uint64()
    _lib.check(_lib.lib().pd_request_device_bytes(None, C.byref(r), 0, C.byref(got)), None)
    assert got.value <= ceiling
