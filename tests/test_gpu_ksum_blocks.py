"""The T=0 Omega integrand (1/Nk) sum_k ln|det(1 + (Hloc - H_k) G'(iw))| against
numpy's determinants on the solver's own G'(iw), for every way the GPU splits
the matrices: spin blocks of 1 to 16 orbitals (one, two and four lanes a
matrix), one joint block where H_k couples the spins, k-points in conjugate
pairs (weights 1 and 2) and unpaired, frequencies on both sides of the change
of form at w = 10 and of the elimination without pivoting, with and without a
bath.  numpy's error is about N^2 eps on a value that may be as small as 1e-8:
2e-13 absolute, 1e-11 relative."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


def _coupled():
    """BHZ with a spin-flip term in H_k: the two 8-orbital spin blocks are one."""
    pt = clusters.bhz(mass=2.1, delta=0.1, nk1=3, ngfiter=20, omega_nodes=16)
    for i in range(4):
        pt.Hk[i, i, 0, 1, 0, 0, :] += 0.2
        pt.Hk[i, i, 1, 0, 0, 0, :] += 0.2
    return pt


def _chain(n, **kw):
    return clusters.chain1d(tprime=1.1, nlat=n, nk=5, ngfiter=20, omega_nodes=16, **kw)


MODELS = {
    "atom": lambda: clusters.square(nx=1, ny=1, maf=0.1, nspin=2, nkx=3, nky=2, ngfiter=5, omega_nodes=16),
    "chain2": lambda: _chain(2),
    "chain3": lambda: _chain(3),
    "square3x2": lambda: clusters.square(nx=3, ny=2, maf=0.1, cdw=0.03, nspin=2, nkx=5, nky=3, ngfiter=30,
                                         omega_nodes=16),
    "bhz": lambda: clusters.bhz(mass=2.1, delta=0.1, nk1=7, ngfiter=20, omega_nodes=16),
    "square3x3": lambda: clusters.square(nx=3, ny=3, maf=0.1, cdw=0.03, nspin=2, nkx=12, nky=11, ngfiter=10,
                                         omega_nodes=16),
    "square5x2": lambda: clusters.square(nx=5, ny=2, cdw=0.03, nspin=1, nkx=3, nky=3, ngfiter=5, omega_nodes=16),
    "square11x1": lambda: clusters.square(nx=11, ny=1, cdw=0.03, nspin=1, nkx=3, nky=3, ngfiter=3, omega_nodes=16),
    "square4x3": lambda: clusters.square(nx=4, ny=3, cdw=0.03, nspin=1, nkx=3, nky=3, ngfiter=3, omega_nodes=16),
    "coupled16": _coupled,
    "bath": lambda: clusters.square_bath(nb=3, nk1=5, ngfiter=30, omega_nodes=16),
}


@pytest.mark.parametrize("name", list(MODELS))
def test_integrand_matches_numpy(name):
    pt = MODELS[name]()
    c = pt.cfg
    s = VcaSolver(c, pt.bath_h, pt.bath_v)
    s.solve(pt.Hloc, pt.Hk, pt.bath_h, pt.bath_v)
    w = np.array([1e-3, 0.3, 2.0, 9.9, 10.1, 40.0, 1e3, 1e5])
    f = s.sum_kmesh(w)
    g = np.moveaxis(clusters.nnn2lso(s.gf_cluster(1j * w)), -1, 0)
    s.close()
    hl, hk = clusters.nnn2lso(pt.Hloc), np.moveaxis(clusters.nnn2lso(pt.Hk), -1, 0)
    n = hl.shape[0]
    p = np.broadcast_to(hl, (len(w), n, n)).copy()
    if pt.bath_h is not None:  # Delta(iw) = V (iw + xmu - h)^-1 V^+
        h, v = pt.bath_h[:, :, 0, 0, 0, 0], pt.bath_v[:, :, 0, 0, 0, 0]
        for i, x in enumerate(w):
            p[i] += v @ np.linalg.inv((1j * x + c.xmu) * np.eye(len(h)) - h) @ v.conj().T
    ref = np.array([np.linalg.slogdet(np.eye(n) + (p[i] - hk) @ g[i])[1].mean() for i in range(len(w))])
    np.testing.assert_allclose(f, ref, rtol=1e-11, atol=2e-13)
