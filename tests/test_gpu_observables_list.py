"""Observables of a thermal list whose states take several fills of the workspace
that their partial sums share: a state of a sector (n_up, n_dw) adds its weight
times n_up to the sum of dens_up over the sites and times n_dw to that of
dens_dw, whatever the state is.

Tolerance: a state's norm is 1 to 1e-12 (2^-F rounding of its elements, or that
of the normalisation), the sums have up to 40 terms: 1e-10."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


# 4x2: 480 partials a state at most, 17 such states a fill; 2x2: all in one
@pytest.mark.parametrize("nx,arith,least", [(4, 0, 40), (4, 1, 40), (2, 0, 10)])
def test_site_sums_of_the_listed_states(nx, arith, least):
    beta = 0.5
    pt = clusters.square(nx=nx, ny=2, U=3.0, xmu=1.2, maf=0.2, cdw=0.1, nspin=2, nkx=1, nky=1, ngfiter=4,
                         omega_nodes=16, contour_nodes=4, lanc_nstates_total=60, beta=beta, bandwidth=8.0, arith=arith)
    s = VcaSolver(pt.cfg)
    s.solve(pt.Hloc, pt.Hk)
    states, zeta, obs = s.states(), s.thermal()["zeta"], s.observables()
    e = np.array([x[1] for x in states])
    w = np.exp(-beta * (e - e.min())) / zeta
    n = np.array([s.sector_info(x[0])[:2] for x in states])
    s.close()
    assert len(states) >= least
    np.testing.assert_allclose(obs["dens_up"].sum(), w @ n[:, 0], rtol=1e-10)
    np.testing.assert_allclose(obs["dens_dw"].sum(), w @ n[:, 1], rtol=1e-10)
    np.testing.assert_allclose(obs["mag"], obs["dens_up"] - obs["dens_dw"], atol=1e-12)
    np.testing.assert_allclose(obs["dens"], obs["dens_up"] + obs["dens_dw"], atol=1e-12)
