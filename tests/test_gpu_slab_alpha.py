"""alpha = <x, H x> of the slab-pair column form: the sums are whole numbers of 128
bits, so they equal Python's, rounded once, at spin spaces of one and several down
configurations, odd row chunks and the largest up space of sixteen sites."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndw,m", [(8, 1, 16), (8, 2, 8), (5, 2, 24), (7, 3, 16), (8, 3, 8)])
def test_alpha_is_the_exact_sum(nup, ndw, m):
    import torch
    pt = clusters.square(nx=4, ny=4, cdw=0.1, nspin=1, nkx=2, nky=2, ngfiter=4, omega_nodes=16)
    s = VcaSolver(pt.cfg)
    s.set_hamiltonian(pt.Hloc)
    isec = next(i for i in range(1, 17 * 17 + 1) if tuple(s.sector_info(i)[:2]) == (nup, ndw))
    _, _, du, dd = s.sector_info(isec)
    fx, f, g = s.arith_info()
    assert fx
    d = du * dd
    x = np.random.default_rng(nup + ndw).normal(size=(m // 8, d, 8))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    xi = np.rint(x * 2.0 ** f).astype(np.int64)
    dx = torch.from_numpy(xi).cuda()
    dy = torch.zeros_like(dx)
    al = torch.zeros(m, dtype=torch.float64, device="cuda")
    s.hxv_alpha_noalloc(isec, dx.data_ptr(), dy.data_ptr(), m, al.data_ptr())
    s.synchronize()
    y = dy.cpu().numpy()
    got = al.cpu().numpy()
    for c in range(0, m, 5):
        total = sum(a * b for a, b in zip(xi[c // 8, :, c % 8].tolist(), y[c // 8, :, c % 8].tolist()))
        want = total / 2 ** (f + g)  # correctly rounded
        # the 128-bit sum becomes a double in one or two roundings
        assert abs(got[c] - want) <= 2 * np.spacing(abs(want)), (c, got[c], want)
    s.close()
