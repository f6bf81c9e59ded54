"""Resident chains on a device short of memory: their scratch (82 MB for the 3x3
cluster's two-spin chains on one state, 2 GB on the 26 states of a thermal list)
is taken for as many chains at a time as fit, in one launch after the other.
The chains are independent and in whole-number arithmetic: equal bit for bit."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaError, VcaSolver

pytestmark = pytest.mark.gpu

THERMAL = dict(lanc_nstates_total=8, beta=1.0, bandwidth=8.0, contour_nodes=4)


def _solve(limit, **kw):
    pt = clusters.square(nx=3, ny=3, maf=0.15, cdw=0.03, nspin=2, nkx=2, nky=2, ngfiter=30, omega_nodes=64, **kw)
    s = VcaSolver(pt.cfg)
    s.set_memory_limit(limit)
    try:
        om = s.solve(pt.Hloc, pt.Hk)
        s.set_memory_limit(0)
        return om, s.states(), s.gf_cluster(np.array([0.05j, 0.7j, 3.0 + 0.5j]))
    finally:
        s.close()


@pytest.mark.parametrize("mb,kw", [(24, {}), (64, {}), (64, THERMAL), (320, THERMAL)])
def test_chains_run_in_what_memory_there_is(mb, kw):
    a, b = _solve(mb << 20, **kw), _solve(0, **kw)
    assert a[0] == b[0] and a[1] == b[1]
    np.testing.assert_array_equal(a[2], b[2])


def test_what_needs_more_is_refused():
    with pytest.raises(VcaError) as e:
        _solve(1 << 20)
    assert e.value.code == -8
    _solve(0)
