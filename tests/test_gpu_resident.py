"""The resident Lanczos runs (whole searches and chains in one launch) against
the separate launches (sector_at_a_time: one sector's search after the other;
two chain streams: the chains as column batches).  The fixed-point sums are
exact and the recurrence is the same, so every result agrees bit for bit.  The
shapes cover one block and clusters of blocks, one and two columns, swapped
spin roles, odd dimensions, two hopping classes, short chains, a search that
exhausts its sector and a cluster with some sectors too large."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


def _two_class(nx, ny, t2, **kw):
    pt = clusters.square(nx=nx, ny=ny, **kw)
    for s in range(pt.cfg.Nspin):  # bonds along y get another magnitude
        for x in range(nx):
            for y in range(ny - 1):
                i, j = clusters.square_site(x, y, nx), clusters.square_site(x, y + 1, nx)
                pt.Hloc[i, j, s, s, 0, 0] = pt.Hloc[j, i, s, s, 0, 0] = t2
    return pt


MODELS = {
    "chain2": lambda: clusters.chain1d(tprime=0.9, nlat=2, nk=4, ngfiter=50, omega_nodes=64),
    "chain4": lambda: clusters.chain1d(tprime=0.9, nlat=4, nk=4, ngfiter=100, omega_nodes=64),
    "chain5": lambda: clusters.chain1d(tprime=1.1, nlat=5, nk=4, ngfiter=60, omega_nodes=64),
    "square2x2": lambda: clusters.square(nx=2, ny=2, maf=0.2, cdw=0.05, nspin=2, nkx=2, nky=2, ngfiter=80,
                                         omega_nodes=64),
    "square3x2_sym": lambda: clusters.square(nx=3, ny=2, maf=0.1, cdw=0.05, nspin=2, nkx=2, nky=2, ngfiter=90,
                                             omega_nodes=64, vca_gf_symmetric=1),
    "two_class3x2": lambda: _two_class(3, 2, -0.7, maf=0.1, nspin=2, nkx=2, nky=2, ngfiter=60, omega_nodes=64),
    "two_class4x2": lambda: _two_class(4, 2, 0.6, maf=0.1, nspin=2, nkx=2, nky=2, ngfiter=40, omega_nodes=64),
    "square4x2": lambda: clusters.square(nx=4, ny=2, maf=0.1, nspin=2, nkx=2, nky=2, ngfiter=40, omega_nodes=64),
    "square3x3": lambda: clusters.square(nx=3, ny=3, maf=0.15, cdw=0.03, nspin=2, nkx=2, nky=2, ngfiter=30,
                                         omega_nodes=64),
    "square3x3_thermal": lambda: clusters.square(nx=3, ny=3, maf=0.15, cdw=0.03, nspin=2, nkx=2, nky=2, ngfiter=30,
                                                 omega_nodes=64, lanc_nstates_total=2, beta=20.0, bandwidth=8.0),
    "square5x2": lambda: clusters.square(nx=5, ny=2, maf=0.1, nspin=1, nkx=2, nky=2, ngfiter=10, omega_nodes=32),
}


def _solve(pt, separate):
    cfg = pt.cfg.copy()
    cfg.sector_at_a_time = separate
    s = VcaSolver(cfg)
    s.set_chain_streams(2 if separate else 1)
    om = s.solve(pt.Hloc, pt.Hk)
    z = np.array([0.05j, 0.7j, 3.0 + 0.5j, 40.0j])
    out = {"omega": om, "sectors": s.sector_energies(), "states": s.states(), "g": s.gf_cluster(z),
           **s.observables()}
    s.close()
    return out


@pytest.mark.parametrize("name", list(MODELS))
def test_resident_runs_equal_separate_launches(name):
    pt = MODELS[name]()
    a, b = _solve(pt, 0), _solve(pt, 1)
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


# FP64: the sums of a dot product run in another order (1e-16 a sum); over a few
# dozen steps and at distance 0.05 of the spectrum (a factor 1/0.05^2) that is
# below 1e-9 of G'.  hxv_variant 1 keeps the separate launches.
FP64_MODELS = {
    "square2x2": lambda: clusters.square(nx=2, ny=2, maf=0.2, cdw=0.05, nspin=2, nkx=2, nky=2, ngfiter=80,
                                         omega_nodes=64, arith=1),
    "chain5_sym": lambda: clusters.chain1d(tprime=1.1, nlat=5, nk=4, ngfiter=60, omega_nodes=64, arith=1,
                                           vca_gf_symmetric=1),
    "bath2": lambda: clusters.square_bath(nb=2, nk1=2, ngfiter=60, omega_nodes=64),
    "bath5": lambda: clusters.square_bath(nb=5, nk1=2, ngfiter=30, omega_nodes=64),
    "bhz": lambda: clusters.bhz(mass=2.2, delta=0.1, nk1=2, ngfiter=40, omega_nodes=64),
    "bhz_phase": lambda: _turned(clusters.bhz(mass=1.8, delta=0.15, nk1=2, ngfiter=30, omega_nodes=64)),
}


def _turned(pt):
    """The same cluster with a gauge phase on one orbital: amplitudes with both parts."""
    ph = np.exp(0.6j)
    pt.Hloc[0, 1:, :, :, 0, :] *= ph
    pt.Hloc[1:, 0, :, :, :, 0] *= np.conj(ph)
    pt.Hloc[0, 0, :, :, 0, 1] *= ph
    pt.Hloc[0, 0, :, :, 1, 0] *= np.conj(ph)
    return pt


@pytest.mark.parametrize("name", list(FP64_MODELS))
def test_resident_fp64_runs_equal_separate_launches(name):
    pt = FP64_MODELS[name]()
    out = []
    for variant in (0, 1):
        cfg = pt.cfg.copy()
        cfg.hxv_variant = variant
        s = VcaSolver(cfg, pt.bath_h, pt.bath_v)
        om = s.solve(pt.Hloc, pt.Hk, pt.bath_h, pt.bath_v)
        out.append((om, s.sector_energies(), [x[0] for x in s.states()],
                    s.gf_cluster(np.array([0.05j, 0.7j, 40.0j])), s.observables()))
        s.close()
    (om, e, st, g, obs), (om1, e1, st1, g1, obs1) = out
    assert sorted(st) == sorted(st1)  # (the order within a degenerate level is rounding)
    np.testing.assert_allclose(e, e1, rtol=1e-12, atol=1e-12)
    np.testing.assert_allclose(g, g1, rtol=0, atol=1e-9 * np.abs(g1).max())
    assert abs(om - om1) <= 1e-10 * abs(om1)
    for k in obs:
        np.testing.assert_allclose(obs[k], obs1[k], rtol=0, atol=1e-10)
