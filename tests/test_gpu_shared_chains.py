"""Channels of (i,j) and (j,i) share a Green's-function chain where their start
vectors agree up to a phase (and, on a real Hamiltonian, complex conjugation).
Every channel of both orders is compared with the oracle, which runs each one
by itself: pole sums off the real axis to 1e-8, the tolerance of the channel
parity test, and the excitation counts exactly."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

MODELS = {
    "real_fixed": lambda **k: clusters.square(nx=2, ny=2, U=8.0, xmu=4.0, maf=0.2, cdw=0.05, nspin=2, nkx=2, nky=2,
                                              ngfiter=80, omega_nodes=64, **k),
    "real_fp64": lambda **k: clusters.square(nx=2, ny=2, U=8.0, xmu=4.0, maf=0.2, cdw=0.05, nspin=2, nkx=2, nky=2,
                                             ngfiter=80, omega_nodes=64, arith=1, **k),
    "complex": lambda **k: clusters.bhz(mass=2.2, delta=0.1, nk1=2, ngfiter=60, omega_nodes=64, **k),
}


@pytest.mark.parametrize("model", list(MODELS))
@pytest.mark.parametrize("symmetric", [0, 1])
def test_both_orders_match_oracle(model, symmetric):
    pt = MODELS[model](vca_gf_symmetric=symmetric)
    c = pt.cfg
    s = VcaSolver(c)
    s.solve(pt.Hloc, pt.Hk)
    o = Oracle.from_point(pt)
    o.solve()
    z = np.array([0.3 + 0.2j, -1.0 + 1.0j, 2.0 + 5.0j])

    def psum(p, w):
        return (w[None, :] / (z[:, None] - p[None, :].real)).sum(axis=1)

    orbs = [(il, io) for il in (1, 2, 4) for io in range(1, c.Norb + 1)]
    for a, b in [(x, y) for x in orbs for y in orbs if x != y]:
        for spin in range(1, c.Nspin + 1):
            for chan in ((1, 2) if symmetric else (1, 2, 3, 4)):
                p, w = s.gf_channel(a[0], b[0], spin, a[1], b[1], 1, chan)
                rp, rw = o.gf_channel(a[0], b[0], spin, a[1], b[1], 0, chan)[:2]
                assert len(p) == len(rp) > 0
                assert np.abs(psum(p, w) - psum(rp, rw)).max() < 1e-8
    s.close()
