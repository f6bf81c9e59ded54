"""The batched search over spin-mirrored points: half-filled and doped (ground
states in a mirrored pair of sectors), screened and not, against plain solves."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("no_screen", [0, 1])
@pytest.mark.parametrize("mu", [2.0, 0.9, 0.2])
def test_batched_omega_matches_plain_solves(mu, no_screen):
    pts = [clusters.square_bath(s_h=h, mu_prime=mu, nb=3, nk1=2, ngfiter=30, omega_nodes=64) for h in (0.8, 1.0, 1.3)]
    cfg = pts[0].cfg.copy()
    cfg.no_sector_screen = no_screen
    s = VcaSolver(cfg, pts[0].bath_h, pts[0].bath_v)

    def stack(xs):
        return np.asfortranarray(np.stack(xs, axis=-1))

    om = s.solve_batch(stack([p.Hloc for p in pts]), pts[0].Hk, stack([p.bath_h for p in pts]),
                       stack([p.bath_v for p in pts]))
    s.close()
    for p, o in zip(pts, om):
        r = VcaSolver(p.cfg, p.bath_h, p.bath_v)
        want = r.solve(p.Hloc, pts[0].Hk, p.bath_h, p.bath_v)
        r.close()
        assert abs(o - want) <= 1e-10 * abs(want), (mu, o, want)
