"""Ground-state vectors from the batched search's own tridiagonal, for sectors that do
not run resident (hxv_variant 1 keeps all of them apart), against a search of
the sector by itself: bit for bit in whole-number arithmetic; in FP64, where the dot
products sum in another order, observables to 1e-10 and energies to 1e-12."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu

SMALL = dict(nkx=2, nky=2, ngfiter=15, omega_nodes=16)
MODELS = {
    "atom": (0, lambda: clusters.square(nx=1, ny=1, xmu=1.3, nspin=1, **SMALL)),  # sectors of one row
    "square2x2": (0, lambda: clusters.square(nx=2, ny=2, maf=0.1, cdw=0.05, nspin=2, **SMALL)),
    "square3x2_doped": (0, lambda: clusters.square(nx=3, ny=2, xmu=0.4, cdw=0.05, nspin=1, **SMALL)),
    "square5x2": (0, lambda: clusters.square(nx=5, ny=2, xmu=0.7, cdw=0.05, nspin=1, **SMALL)),
    "square3x2_fp64": (1, lambda: clusters.square(nx=3, ny=2, maf=0.1, cdw=0.05, nspin=2, arith=1, **SMALL)),
    "bath5": (1, lambda: clusters.square_bath(nb=5, nk1=2, ngfiter=15, omega_nodes=16)),
    "bhz": (1, lambda: clusters.bhz(mass=2.2, delta=0.1, nk1=2, ngfiter=15, omega_nodes=16)),
}


def _solve(pt, niter, one_by_one):
    cfg = pt.cfg.copy()
    cfg.hxv_variant, cfg.lanc_niter, cfg.sector_at_a_time = 1, niter, one_by_one
    s = VcaSolver(cfg, pt.bath_h, pt.bath_v)
    s.solve(pt.Hloc, pt.Hk, pt.bath_h, pt.bath_v)
    out = [x[0] for x in s.states()], np.array([x[1] for x in s.states()]), s.observables(), s.gf_cluster([0.5j, 9.0j])
    s.close()
    return out


@pytest.mark.parametrize("niter", [7, 512])  # unconverged and converged searches
@pytest.mark.parametrize("name", list(MODELS))
def test_vectors_match_a_search_by_itself(name, niter):
    fp64, make = MODELS[name]
    if fp64 and niter == 7:
        niter = 512  # two unconverged FP64 runs agree as their rounding does
    pt = make()
    a, b = _solve(pt, niter, 0), _solve(pt, niter, 1)
    if not fp64:
        assert a[0] == b[0]
        np.testing.assert_array_equal(a[1], b[1])
        np.testing.assert_array_equal(a[3], b[3])
    else:
        assert sorted(a[0]) == sorted(b[0])
        np.testing.assert_allclose(a[1], b[1], rtol=1e-12)
        np.testing.assert_allclose(a[3], b[3], rtol=0, atol=1e-9)
    for k in a[2]:
        np.testing.assert_allclose(a[2][k], b[2][k], rtol=0, atol=1e-10 if fp64 else 0)
