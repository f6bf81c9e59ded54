"""The two forms of the T=0 Omega integrand on both sides of the line between them
(2^15 determinants a call): the calls next to the line agree with the smallest
one, and only the one above it launches the transposition that whole
determinants per thread read.

Tolerance as in test_gpu_ksum_blocks.py, whose models these are: each form is
within N^2 eps of the value, which may be as small as 1e-8."""
import numpy as np
import pytest

from test_gpu_ksum_blocks import MODELS
from vca_gb300.solver import VcaSolver, pair_kpoints

pytestmark = pytest.mark.gpu

W = np.array([1e-3, 0.3, 2.0, 9.9, 10.1, 40.0, 1e3, 1e5])


@pytest.mark.parametrize("name", list(MODELS))
def test_both_sides_of_the_line(name):
    pt = MODELS[name]()
    c = pt.cfg
    s = VcaSolver(c, pt.bath_h, pt.bath_v)
    s.solve(pt.Hloc, pt.Hk, pt.bath_h, pt.bath_v)
    paired = not np.any(pt.Hloc.imag) and name != "coupled16"
    nk = len(pair_kpoints(pt.Hk)[0]) if paired else pt.Nk
    blocks = 1 if name == "coupled16" else c.Nspin
    line = -(-(1 << 15) // (nk * blocks))
    few = s.sum_kmesh(W)
    launches = []
    for n in (line - 1, line):
        w = np.resize(W, n)
        s.sum_kmesh(w)
        before = s.kernel_launches()
        f = s.sum_kmesh(w)
        launches.append(s.kernel_launches() - before)
        np.testing.assert_allclose(f, np.resize(few, n), rtol=1e-11, atol=2e-13)
    s.close()
    assert launches[1] == launches[0] + 1
