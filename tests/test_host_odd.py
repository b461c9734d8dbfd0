"""Host-buffer solves of odd batches equal the device solve bit for bit: the chunks, even
ones but for the last, take the cut of a system into sub-segments that the odd batch does
(16- and 32-row ones, any-length periodic ones, clusters, short segments)."""
import numpy as np
import pytest

from filtered_tdma_b200 import Solver
from filtered_tdma_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sys,n_row,P,cyclic", [
    (8001, 48, 2, False), (9601, 48, 4, False), (8193, 64, 4, False), (9001, 250, 8, False),
    (8193, 512, 8, False), (5001, 1024, 16, False), (8193, 7, 2, False),
    (9001, 85, 4, True), (8193, 192, 4, True), (8193, 256, 4, True), (8193, 64, 4, True),
    (4801, 700, 8, True)])
def test_odd_host_batches_equal_the_device_solve(cuda, n_sys, n_row, P, cyclic):
    import torch
    arrays = [torch.from_numpy(v) for v in W.row_varying(n_sys, n_row, seed=n_row)]
    s = Solver("pascal", n_sys, n_row, P)
    dev = [v.to(cuda) for v in arrays]
    X = torch.empty_like(dev[3])
    s.solve_out(*dev, X, cyclic=cyclic)
    host = torch.full_like(arrays[3], 7.0).pin_memory()
    s.solve_host(*[v.pin_memory() for v in arrays], host, cyclic=cyclic)
    torch.cuda.synchronize()
    assert np.array_equal(host.numpy(), X.cpu().numpy())
    assert s.status() == 0
