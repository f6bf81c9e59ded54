"""The T=0 Omega integrand on meshes whose threads sum many determinants: from
1,216 frequencies a call on, every k of a node lies in one block.  Above w = 10
the determinants are eliminated without pivoting and close to 1; a uniform field
on the cluster makes their logarithms add up with one sign, so the product over
a thread's k runs far below or above 1.  Reference: numpy's determinants, one by
one, on the solver's own G'.

Tolerance: an elimination of n <= 12 rows and numpy's are each within n^2 eps of
ln|det| (3e-14), and a running sum of m <= 4,000 logarithms whose total is at
most m |f| adds m eps |f| / 2: with |f| < 0.4 below 2e-13 of the mean."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu

W = np.array([9.9, 10.05, 12.0, 15.0, 40.0, 1e3])


def _square(nx, ny, nk, nspin=1, **kw):
    return clusters.square(nx=nx, ny=ny, nspin=nspin, nkx=nk, nky=nk, ngfiter=20, omega_nodes=16, **kw)


MODELS = {
    "atom": lambda: _square(1, 1, 256, U=0.0, xmu=2.0, mu_shift=-1.5),
    "2x2 small det": lambda: _square(2, 2, 192, U=0.0, xmu=4.0, mu_shift=1.0),
    "2x2 large det": lambda: _square(2, 2, 192, U=0.0, xmu=4.0, mu_shift=-1.0),
    "3x3 two spins": lambda: _square(3, 3, 128, nspin=2, U=0.0, xmu=-2.4, mu_shift=0.5),
    "3x3 two spins, up": lambda: _square(3, 3, 128, nspin=2, U=0.0, xmu=-2.4, mu_shift=-0.5),
    "4x3 half filled": lambda: _square(4, 3, 320),
    "chain2": lambda: clusters.chain1d(nlat=2, nk=60000, xmu=3.0, ngfiter=20, omega_nodes=16),
    "bath": lambda: clusters.square_bath(nb=2, nk1=128, mu_prime=3.0, ngfiter=20, omega_nodes=16),
}


@pytest.mark.parametrize("name", list(MODELS))
def test_many_determinants_a_thread(name):
    pt = MODELS[name]()
    c = pt.cfg
    s = VcaSolver(c, pt.bath_h, pt.bath_v)
    s.solve(pt.Hloc, pt.Hk, pt.bath_h, pt.bath_v)
    f = s.sum_kmesh(np.tile(W, 203)).reshape(203, len(W))
    g = np.moveaxis(clusters.nnn2lso(s.gf_cluster(1j * W)), -1, 0)
    s.close()
    hl, hk = clusters.nnn2lso(pt.Hloc), np.moveaxis(clusters.nnn2lso(pt.Hk), -1, 0)
    n = hl.shape[0]
    ref = np.zeros(len(W))
    for i, w in enumerate(W):
        p = hl
        if pt.bath_h is not None:  # Delta(iw) = V (iw + xmu - h)^-1 V^+
            h, v = pt.bath_h[:, :, 0, 0, 0, 0], pt.bath_v[:, :, 0, 0, 0, 0]
            p = hl + v @ np.linalg.inv((1j * w + c.xmu) * np.eye(len(h)) - h) @ v.conj().T
        nb = n // c.Nspin
        for b in range(0, n, nb):  # H and G' are diagonal in the spin
            q = slice(b, b + nb)
            ref[i] += np.concatenate([np.linalg.slogdet(np.eye(nb) + (p[q, q] - h[:, q, q]) @ g[i, q, q])[1]
                                      for h in np.array_split(hk, 64)]).mean()
    np.testing.assert_array_equal(f, f[:1].repeat(203, axis=0))
    np.testing.assert_allclose(f[0], ref, rtol=0, atol=2e-13)
