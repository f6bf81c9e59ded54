"""G' and the grids in the caller's index order, re-ordered on the device in pieces:
many points at once (more than one piece of 16 MB, the last one short) against
the same points a few at a time, two orbitals and two spins, and a single site."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n", [("bhz", 9001), ("square3x2", 7300), ("site", 20), ("site", 1)])
def test_many_points_equal_few_at_a_time(name, n):
    small = dict(ngfiter=10, omega_nodes=16)
    pt = {"bhz": lambda: clusters.bhz(mass=2.2, delta=0.1, nk1=2, **small),
          "square3x2": lambda: clusters.square(nx=3, ny=2, maf=0.1, nspin=2, nkx=2, nky=2, **small),
          "site": lambda: clusters.square(nx=1, ny=1, nspin=1, nkx=2, nky=2, **small)}[name]()
    s = VcaSolver(pt.cfg)
    s.solve(pt.Hloc, pt.Hk)
    z = 1j * np.linspace(0.1, 50.0, n)
    g = s.gf_cluster(z)
    for at in (0, n // 2, max(0, n - 3)):
        np.testing.assert_array_equal(g[..., at:at + 3], s.gf_cluster(z[at:at + 3]))
    s.close()
