"""The wide solve's general form (tails, odd batches, clusters) and the periodic
any-length solve, through the default dispatch.

Sizes at the edges of their ranges: tails of 1, 2, 31 and 32 rows, odd n_sys (rows
in pairs, an unpaired last row), one sub-segment to eight CTAs a system, group
widths down to the narrowest, last groups partly outside the batch.  Bar: the
tiled path's 1e-12 relative to the serial Thomas, on coefficients that differ in
every row and system.  The entries a non-periodic system does not use (A of the
first row, C of the last) hold NaN where the segment kernels took the shape
before, which ignore them.
"""
import numpy as np
import pytest

from filtered_tdma_b200 import Solver
from filtered_tdma_b200 import _lib as L
from filtered_tdma_b200 import workloads as W

pytestmark = pytest.mark.gpu


def check(cuda, orc, n_sys, n_row, P, cyclic=False, dt=np.float64, nan=False):
    import torch
    A, B, C, D = [np.ascontiguousarray(v, dtype=dt)
                  for v in W.row_varying(n_sys, n_row, seed=n_sys + 7 * n_row)]
    wid = [v.astype(np.float64) for v in (A, B, C, D)]
    ref = orc.thomas_cyclic(*wid) if cyclic else orc.thomas(*wid)
    if nan:
        A[0] = np.nan
        C[-1] = np.nan
    dev = [torch.from_numpy(v).to(cuda) for v in (A, B, C, D)]
    # one row more than the solution: nothing is written past it
    X = torch.full((n_row + 1, n_sys), 7.0, dtype=torch.float64, device=cuda)
    s = Solver("pascal", n_sys, n_row, P,
               precision=L.FP64 if dt == np.float64 else L.FP32_STORE)
    f = s.solve_out if dt == np.float64 else s.solve_f32
    f(*dev, X, n_sys=n_sys, n_row=n_row, cyclic=cyclic)
    x = X.cpu().numpy()
    assert np.max(np.abs(x[:-1] - ref)) <= 1e-12 * np.max(np.abs(ref))
    assert (x[-1] == 7.0).all()
    assert s.status() == 0
    if dt == np.float64:  # in place
        s.solve(*dev, n_sys=n_sys, n_row=n_row, cyclic=cyclic)
        assert np.array_equal(dev[3].cpu().numpy(), x[:-1])


@pytest.mark.parametrize("n_row", [33, 34, 35, 63, 65, 95, 97, 129, 250, 481, 511])
@pytest.mark.parametrize("n_sys", [301, 5002, 20001])
def test_tails(cuda, orc, n_sys, n_row):
    check(cuda, orc, n_sys, n_row, 2 if n_row <= 128 else 8, nan=True)


@pytest.mark.parametrize("n_sys,n_row", [(301, 32), (9601, 64), (5003, 320), (4999, 512),
                                         (37, 20), (20003, 7)])
def test_odd_batches(cuda, orc, n_sys, n_row):
    check(cuda, orc, n_sys, n_row, 2 if n_row <= 128 else 8, nan=True)


@pytest.mark.parametrize("n_sys,n_row", [(3000, 48), (66000, 48), (9600, 176), (4800, 272),
                                         (4800, 496)])
@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_row_counts_of_the_narrow_kernel(cuda, orc, n_sys, n_row, dt):
    check(cuda, orc, n_sys, n_row, 2, dt=dt)


@pytest.mark.parametrize("n_sys,n_row", [(2402, 513), (2401, 545), (1202, 700), (2400, 1024),
                                         (1201, 1025), (601, 2047), (300, 3000), (98, 4096),
                                         (603, 2063)])
def test_clusters(cuda, orc, n_sys, n_row):
    check(cuda, orc, n_sys, n_row, 16, nan=n_row % 16 != 0 and n_row < 4096)


def test_clusters_fp32(cuda, orc):
    check(cuda, orc, 2400, 1088, 8, dt=np.float32)


@pytest.mark.parametrize("n_sys,n_row", [
    (301, 32), (3001, 128), (1003, 512),          # one CTA, odd n_sys
    (2400, 1024), (1201, 1536), (300, 4096),      # whole sub-segments over a cluster
    (1000, 192), (1001, 85), (4100, 85), (1000, 481), (38, 21),  # any length, one CTA
    (600, 1537), (601, 1537), (602, 700),         # any length, clusters
])
def test_periodic(cuda, orc, n_sys, n_row):
    check(cuda, orc, n_sys, n_row, 6 if n_row < 512 else 16, cyclic=True)
