"""The self profiles of a lattice set come from exact pair counts in FP64, whatever form
the other pairs are summed in: an FP32 request's excluded-volume and hydration
profiles of grid dummies are the double-precision ones.

Tolerance 1e-12 of a point, as stated for the counts (the FP64 form that they are
compared with is good to 1e-14; the sums over the counts run over a few thousand
bins, of which a point at its minimum is 1e-4)."""
import numpy as np
import pytest

from conftest import term_errors
from pripps_b200 import workloads
from pripps_b200.debye import solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spacing,nq,qmax", [(60, 1.2, 40, 0.5), (900, 1.5, 120, 0.6),
                                               (2500, 1.5, 250, 0.5)])
def test_lattice_self_profiles_are_exact(gpu_ctx, n, spacing, nq, qmax):
    g = workloads.small_globule(n, 3).globule
    got = solve(workloads.grid_solvent_request(g, 0.0, qmax, nq, "fp32", spacing), gpu_ctx)
    ref = workloads.grid_solvent_request(g, 0.0, qmax, nq, "fp64", spacing)
    assert len(ref.lattices) == 2
    ref.lattices = None
    err = term_errors(got, solve(ref, gpu_ctx))
    assert np.all(err < 1e-5) and np.all(err[1:3] < 1e-12), err


def test_lattice_point_off_its_grid_in_every_form(gpu_ctx):
    """A point moved off its lattice is refused where the other pairs are directions
    and where they are pairs."""
    from pripps_b200.errors import ValidationError
    for n, qmax in ((900, 0.5), (30, 0.5), (300, 6.0)):
        req = workloads.grid_solvent_request(workloads.small_globule(n, 3).globule, 0.0, qmax, 30,
                                             "fp32", 1.6)
        k = int(np.flatnonzero(req.species == req.lattices[0][0])[3])
        req.xyz = req.xyz.copy()
        req.xyz[k, 1] += 0.05
        with pytest.raises(ValidationError):
            solve(req, gpu_ctx)
