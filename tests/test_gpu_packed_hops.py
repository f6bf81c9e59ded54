"""The column H x v with packed up hops (one amplitude class, up spaces of 128
to 1023 configurations, rows in hop-count order) against the staged form on the
same columns in natural order: exact sums and one rounding in both, so Y agrees
bit for bit, and alpha with it.  Sectors cover both ends of the range, row
counts that are no multiple of 16, one to several slabs, a last slab of 8
columns, and spin roles of different sizes."""
import numpy as np
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu

SECTORS = [  # cluster, (n_up, n_dw), columns
    ((5, 2), (5, 5), 16), ((5, 2), (4, 5), 24), ((5, 2), (6, 3), 40),
    ((4, 3), (3, 2), 16), ((4, 3), (4, 3), 24), ((4, 3), (5, 1), 32), ((4, 3), (6, 2), 16), ((4, 3), (7, 6), 16),
]


@pytest.mark.parametrize("shape,filling,m", SECTORS)
def test_packed_equals_staged(shape, filling, m):
    import torch
    pt = clusters.square(nx=shape[0], ny=shape[1], maf=0.1, nspin=2, nkx=1, nky=1, ngfiter=5, omega_nodes=16)
    ns = shape[0] * shape[1]
    isec = 1 + filling[1] + filling[0] * (ns + 1)
    ys, order = [], None
    for variant in (0, 2):
        cfg = pt.cfg.copy()
        cfg.hxv_variant = variant
        s = VcaSolver(cfg)
        s.set_hamiltonian(pt.Hloc)
        _, _, du, dd = s.sector_info(isec)
        d = du * dd
        fx, scale, _ = s.arith_info()
        assert fx and 128 <= du <= 1023
        x = np.random.default_rng(9).normal(size=(d, m))
        x /= np.linalg.norm(x, axis=0, keepdims=True)
        xi = np.rint(x * 2.0 ** scale).astype(np.int64)
        if variant == 2:
            order = s.sector_row_order(isec)
            xi = xi[order]
        slab = np.ascontiguousarray(xi.reshape(d, m // 8, 8).transpose(1, 0, 2))
        dx = torch.from_numpy(slab).cuda()
        dy = torch.zeros_like(dx)
        al = torch.zeros(m, dtype=torch.float64, device="cuda")
        s.hxv_alpha_noalloc(isec, dx.data_ptr(), dy.data_ptr(), m, al.data_ptr())
        s.synchronize()
        torch.cuda.synchronize()
        y = dy.cpu().numpy().reshape(m // 8, d, 8).transpose(1, 0, 2).reshape(d, m)
        ys.append((y, al.cpu().numpy()))
        s.close()
    np.testing.assert_array_equal(ys[0][0][order], ys[1][0])
    np.testing.assert_array_equal(ys[0][1], ys[1][1])
