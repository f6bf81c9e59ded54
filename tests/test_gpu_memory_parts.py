"""Calls on a device short of memory whose large workspaces are a matter of speed
only: sum_kmesh without room for the transposed M of its whole-determinant form,
G' without room for every chain's value at every point.  Each call has to run in
the memory that its arrays and the smallest call take (found by bisection) and
128 or 256 KB besides.

Tolerance: G' is the same arithmetic point by point, equal bit for bit; the two
forms of the integrand as in test_gpu_ksum_route.py."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaError, VcaSolver

pytestmark = pytest.mark.gpu


@pytest.fixture
def solved():
    pt = clusters.square(nx=2, ny=2, maf=0.2, nspin=2, nkx=64, nky=64, ngfiter=60, omega_nodes=64)
    s = VcaSolver(pt.cfg)
    s.solve(pt.Hloc, pt.Hk)
    yield s
    s.close()


def _least(s, call):
    """Smallest memory limit, in steps of 4 KB, under which the call runs."""
    lo, hi = 0, 1 << 15
    while hi - lo > 1:
        mid = (lo + hi) // 2
        s.set_memory_limit(mid << 12)
        try:
            call()
            hi = mid
        except VcaError as e:
            assert e.code == -8
            lo = mid
    s.set_memory_limit(0)
    return hi << 12


def test_sum_kmesh_without_the_transposed_matrices(solved):
    s = solved
    w = np.array([1e-3, 0.3, 2.0, 9.9, 10.1, 40.0, 1e3, 1e5])  # 8 x 2 x 2,050 determinants: 32,800
    n0 = s.kernel_launches()
    ref = s.sum_kmesh(w)
    n1 = s.kernel_launches()
    s.set_memory_limit(_least(s, lambda: s.sum_kmesh(w[:1])) + (128 << 10))
    n2 = s.kernel_launches()
    f = s.sum_kmesh(w)
    assert s.kernel_launches() - n2 == n1 - n0 - 1  # no transposition
    s.set_memory_limit(0)
    np.testing.assert_allclose(f, ref, rtol=1e-11, atol=2e-13)


def test_gf_in_runs_of_points(solved):
    s = solved
    nz = 4000
    z = 0.1 + 1j * np.linspace(0.05, 40.0, nz)
    ref = s.gf_cluster(z)
    n, nelem = 8, 32
    arrays = 16 * nz * (1 + n * n + nelem)  # z, G', element sums
    s.set_memory_limit(_least(s, lambda: s.gf_cluster(z[:1])) + arrays + (256 << 10))
    g = s.gf_cluster(z)
    s.set_memory_limit(0)
    np.testing.assert_array_equal(g, ref)
