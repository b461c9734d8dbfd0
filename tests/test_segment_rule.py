"""Small batches on both sides of the rule that keeps some of them on the segment kernels
(few segments of at most 16 rows, at most 4096 systems), against the serial Thomas."""
import numpy as np
import pytest

from filtered_tdma_b200 import Solver
from filtered_tdma_b200 import _lib as L
from filtered_tdma_b200 import workloads as W

pytestmark = pytest.mark.gpu

# n_sys, n_row, P, whether the segment kernels keep the non-periodic / the periodic batch
# (their result is then the reference-order one to the bit)
SHAPES = [(4096, 50, 4, True, True), (4098, 50, 4, False, False), (4096, 65, 4, False, False),
          (512, 90, 6, True, True), (512, 50, 8, False, True), (3074, 50, 8, False, False),
          (512, 120, 8, False, True), (300, 250, 16, False, False), (511, 50, 4, False, False)]


@pytest.mark.parametrize("n_sys,n_row,P,seg,seg_cyclic", SHAPES)
@pytest.mark.parametrize("cyclic", [False, True])
def test_rule(cuda, orc, n_sys, n_row, P, seg, seg_cyclic, cyclic):
    import torch
    arrays = W.row_varying(n_sys, n_row, seed=n_sys + n_row)
    dev = [torch.from_numpy(v).to(cuda) for v in arrays]
    X = torch.empty_like(dev[3])
    got = []
    for flags in (0, L.FLAG_REFERENCE_ORDER):
        s = Solver("pascal", n_sys, n_row, P, flags=flags)
        s.solve_out(*dev, X, cyclic=cyclic)
        got.append(X.cpu().numpy())
        assert s.status() == 0
    ref = orc.thomas_cyclic(*arrays) if cyclic else orc.thomas(*arrays)
    assert np.max(np.abs(got[0] - ref)) <= 1e-12 * np.max(np.abs(ref))
    assert np.array_equal(*got) == (seg_cyclic if cyclic else seg)
