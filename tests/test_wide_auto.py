"""The wide tiled kernel where the default dispatch picks it: every group width
it is instantiated for, group counts that are not a power of two, last groups
partly outside the batch, and the 256-thread form of which two share an SM.

Bar: the tiled path's 1e-12 relative to the serial Thomas (FP32 storage: of the
widened values), on batches whose coefficients differ in every row and system.
"""
import numpy as np
import pytest

from filtered_tdma_b200 import Solver
from filtered_tdma_b200 import _lib as L
from filtered_tdma_b200 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [
    (40004, 64, False),    # 256 systems per CTA, 2 sub-segments
    (20000, 64, True),     # 128 systems, 256 threads
    (20004, 96, False),    # 128 systems, 3 sub-segments on 4 lanes
    (9604, 160, False),    # 5 sub-segments on 8 lanes: two passes of the reduced solve
    (10000, 256, True),
    (5000, 416, False),    # 13 sub-segments on 16 lanes
    (5000, 512, False),    # 32 systems, last group of 8
    (2052, 512, False),    # 16 systems, 256 threads
    (300, 512, True),      # 16 systems, few groups
]


@pytest.mark.parametrize("n_sys,n_row,cyclic", SHAPES)
@pytest.mark.parametrize("precision", [L.FP64, L.FP32_STORE])
def test_wide_default_dispatch(cuda, orc, n_sys, n_row, cyclic, precision):
    import torch
    dt = np.float32 if precision == L.FP32_STORE else np.float64
    arrays = [np.ascontiguousarray(v, dtype=dt)
              for v in W.row_varying(n_sys, n_row, seed=n_sys + n_row)]
    dev = [torch.from_numpy(v).to(cuda) for v in arrays]
    X = torch.full((n_row, n_sys), 7.0, dtype=torch.float64, device=cuda)
    s = Solver("pascal", n_sys, n_row, 4, precision=precision)
    f = s.solve_out if precision == L.FP64 else s.solve_f32
    for _ in range(2):  # tensor memory is given back between launches
        f(*dev, X, cyclic=cyclic)
    wid = [v.astype(np.float64) for v in arrays]
    ref = orc.thomas_cyclic(*wid) if cyclic else orc.thomas(*wid)
    assert np.max(np.abs(X.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))
    assert s.status() == 0
