"""Sectors (n_up, n_dw) and (n_dw, n_up) share their lowest energy when the spins
mirror each other: equal one-body parts (Nspin = 1, Nspin = 2 without a spin
field), conjugate ones (BHZ), and not with a field, where all sectors run."""
import numpy as np
import pytest

from oracle.oracle import Oracle
from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu

SMALL = dict(nkx=2, nky=2, ngfiter=20, omega_nodes=16)
MODELS = {
    "equal": lambda: clusters.square(nx=2, ny=2, cdw=0.05, nspin=1, **SMALL),
    "equal_doped": lambda: clusters.square(nx=3, ny=2, xmu=0.4, cdw=0.05, nspin=1, **SMALL),  # odd ground states
    "equal_two_spins": lambda: clusters.square(nx=3, ny=2, xmu=0.4, cdw=0.05, nspin=2, **SMALL),
    "field": lambda: clusters.square(nx=3, ny=2, maf=0.2, cdw=0.05, xmu=0.9, nspin=2, **SMALL),
    "bath_fp64": lambda: clusters.square_bath(nb=3, mu_prime=1.1, nk1=2, ngfiter=20, omega_nodes=16),
    "bhz": lambda: clusters.bhz(mass=2.2, delta=0.1, nk1=2, ngfiter=20, omega_nodes=16),
    "square5x2": lambda: clusters.square(nx=5, ny=2, xmu=0.7, cdw=0.05, nspin=1, **SMALL),
}


def _solve(pt, **kw):
    cfg = pt.cfg.copy()
    for k, v in kw.items():
        setattr(cfg, k, v)
    s = VcaSolver(cfg, pt.bath_h, pt.bath_v)
    s.solve(pt.Hloc, pt.Hk, pt.bath_h, pt.bath_v)
    out = s.sector_energies(), s.states()
    s.close()
    return out


@pytest.mark.parametrize("name", list(MODELS))
def test_sector_energies_and_list_match_the_oracle(name):
    pt = MODELS[name]()
    e, states = _solve(pt)
    o = Oracle.from_point(pt)
    o.solve()
    np.testing.assert_allclose(e, o.sector_energies(), rtol=1e-10, atol=1e-10)
    assert sorted(x[0] for x in states) == sorted(x[0] for x in o.states())


@pytest.mark.parametrize("name", ["equal_doped", "square5x2"])
@pytest.mark.parametrize("niter", [6, 512])
def test_unconverged_sectors_run_their_own_search(name, niter):
    """Six steps converge the smallest sectors only: the others keep the energies of
    their own searches, whole-number arithmetic gives them bit for bit."""
    pt = MODELS[name]()
    a, b = _solve(pt, lanc_niter=niter), _solve(pt, lanc_niter=niter, sector_at_a_time=1)
    np.testing.assert_array_equal(a[0], b[0])
    assert a[1] == b[1]
