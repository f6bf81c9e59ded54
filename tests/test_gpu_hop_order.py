"""Rows of a spin space by decreasing hop count (stable), as the position-ordered
kernels hold them: sizes below, at and above the launch's block of 128 rows and
the 1024-row chunks it compares against."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,fillings", [(2, 2, (0, 1, 2)), (3, 3, (4,)), (4, 3, (2, 4, 5, 6)), (7, 2, (4, 6, 7))])
def test_rows_by_decreasing_hop_count(nx, ny, fillings):
    ns = nx * ny
    pt = clusters.square(nx=nx, ny=ny, nspin=1, nkx=2, nky=2, ngfiter=4, omega_nodes=16)
    s = VcaSolver(pt.cfg)
    s.set_hop_pairing(False)
    s.set_hamiltonian(pt.Hloc)
    h = np.asarray(pt.Hloc).reshape(-1)
    bonds = _bonds(nx, ny)
    assert np.count_nonzero(np.abs(h) > 0) >= len(bonds)
    for n in fillings:
        words = np.array([w for w in range(1 << ns) if bin(w).count("1") == n])
        count = np.zeros(len(words), dtype=int)
        for a, b in bonds:  # a bond moves a particle when one end is filled
            count += ((words >> a) & 1) != ((words >> b) & 1)
        want = np.argsort(-count, kind="stable")
        order = s.sector_row_order(1 + n * (ns + 1))  # ndw = 0: the up space itself
        np.testing.assert_array_equal(order, want)
    s.close()


def _bonds(nx, ny):
    site = lambda x, y: x + nx * y
    return ([(site(x, y), site(x + 1, y)) for x in range(nx - 1) for y in range(ny)] +
            [(site(x, y), site(x, y + 1)) for x in range(nx) for y in range(ny - 1)])
