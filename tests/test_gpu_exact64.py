"""Both routes of the binary64 bond arithmetic against the oracle.

Lengths within 2^+-200 that change by less than a factor of two take their
root and quotients from the integer pipe (``csrc/pp_exact64.cuh``), all
others the binary64 pipe's own operations.  Bit-identical to the oracle on
lattices on either side of each limit: scaled far down or up, bonds
stretched to several times their length or squeezed to a fraction, and
subnormal displacement differences.
"""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.gpu_helpers import lattice, pull_bcs, run_integrator, run_oracle

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]

#: name: (scale of the lattice, face displacement in spacings, pulled axis)
CASES = {"ordinary": (1.0, 1e-3, 0),
         "inside_low": (2.0 ** -196, 1e-3, 0),
         "outside_low": (2.0 ** -204, 1e-3, 0),
         "inside_high": (2.0 ** 196, 1e-3, 0),
         "outside_high": (2.0 ** 204, 1e-3, 0),
         "stretched": (1.0, 5.0, 0),
         "squeezed": (1.0, -0.45, 0),
         "subnormal": (1.0, 1e-309, 1),
         "small": (1.0, 1e-140, 1),
         "tiny": (1.0, 1e-155, 1)}


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("case", sorted(CASES))
def test_bits(case, fused):
    import probabilistic_peridynamics_gb300 as pp
    scale, pull, axis = CASES[case]
    coords, _, _, family, nlist, n_neigh = lattice(6, 5, 4, 1.0)
    n = coords.shape[0]
    bc_types, bc_values = pull_bcs(coords, axis)
    setup = dict(coords=coords * scale, volume=np.ones(n), family=family,
                 nlist=nlist, n_neigh=n_neigh, bc_types=bc_types,
                 bc_values=bc_values,
                 force_bc_types=np.zeros((n, 3), dtype=np.intc),
                 force_bc_values=np.zeros((n, 3)), nnodes=n,
                 max_neigh=nlist.shape[1], k=0.01 * scale,
                 s0=20.0 if case == "stretched" else 0.02, dt=0.5)
    steps = 4
    mags = pull * scale * np.arange(1, steps + 1) / steps
    with np.errstate(all="ignore"):
        ref = run_oracle("euler", setup, steps, mags)
        out = run_integrator(pp.EulerCUDA(dt=0.5, fused=fused), setup, steps,
                             mags)
    for got, want in zip(out, ref):
        assert np.array_equal(got, want, equal_nan=True)
