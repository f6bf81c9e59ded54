"""max_exc from the top of each chain's tridiagonal against the poles' QL.

Both find an eigenvalue of the same matrix, each within n eps |T| (n <= 60 rows,
|T| within the cluster's band, < 40 here): 60 * 2.2e-16 * 40 = 5.3e-13, and as
much again for the other side."""
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ngf", [(1, 1, 8), (2, 1, 50), (2, 2, 1), (2, 2, 60), (3, 2, 33)])
def test_max_exc_matches_the_poles(nx, ny, ngf):
    pt = clusters.square(nx=nx, ny=ny, U=4.0, xmu=1.9, nspin=1, nkx=2, nky=2, ngfiter=ngf, omega_nodes=16)
    cfg = pt.cfg.copy()
    cfg.lanc_nstates_total, cfg.beta, cfg.bandwidth = 2, 6.0, 8.0
    s = VcaSolver(cfg)
    # a state's H x v rounds the same way in every solve, so both have the same chains
    got = []
    for limit in (60, 61):  # any other limit than the default takes the poles
        s.close()
        s = VcaSolver(cfg)
        s.set_ql_max_iter(limit)
        s.solve(pt.Hloc, pt.Hk)
        got.append(s.thermal()["max_exc"])
    s.close()
    assert abs(got[0] - got[1]) < 1.1e-12, got
