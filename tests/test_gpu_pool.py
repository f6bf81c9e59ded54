"""The context's memory pool: bounded between calls (256 MB and what the driver
rounds it up to) and given back when the solver closes."""
import pytest

from vca_gb300 import clusters
from vca_gb300.solver import VcaSolver

pytestmark = pytest.mark.gpu


def test_pool_is_bounded_and_given_back():
    import torch
    mb = 1 << 20
    pt = clusters.square(nx=4, ny=3, cdw=0.03, nspin=1, nkx=2, nky=2, ngfiter=3, omega_nodes=16)
    s = VcaSolver(pt.cfg)  # the CUDA context and its kernels are loaded by the first solve
    s.solve(pt.Hloc, pt.Hk)
    s.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = VcaSolver(pt.cfg)
    for _ in range(3):  # column batches of gigabytes come and go
        s.solve(pt.Hloc, pt.Hk)
        s.synchronize()
        assert before - torch.cuda.mem_get_info()[0] < 400 * mb
    s.close()
    torch.cuda.synchronize()
    assert abs(before - torch.cuda.mem_get_info()[0]) < 64 * mb
