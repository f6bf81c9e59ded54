"""FP64 dot products of one and many columns, from one to 608 partial sums a column:
the FP64 solve (separate launches) against the fixed-point one.  The ground
energies agree to the rounding of a few dozen recurrence steps, 1e-12 relative,
and Green's functions at distance >= 0.7 of the spectrum to 1e-9."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(2, 1), (2, 2), (3, 2), (4, 2), (5, 2)])  # largest sectors 4 .. 63504 rows
def test_fp64_solve_matches_fixed_point(nx, ny):
    pt = clusters.square(nx=nx, ny=ny, cdw=0.05, xmu=3.7, nspin=1, nkx=2, nky=2, ngfiter=25, omega_nodes=16)
    out = []
    for arith in (1, 0):
        cfg = pt.cfg.copy()
        cfg.arith, cfg.hxv_variant = arith, arith  # variant 1 keeps the separate launches
        s = VcaSolver(cfg)
        s.solve(pt.Hloc, pt.Hk)
        out.append((s.energies()[0], s.gf_cluster(np.array([0.7j, 3.0j, 40.0j]))))
        s.close()
    assert abs(out[0][0] - out[1][0]) <= 1e-12 * abs(out[1][0])
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=0, atol=1e-9)
