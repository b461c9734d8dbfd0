"""Pivots at the ends of the FP64 range: row counts that 16 does not divide, odd batches and
periodic lengths that are not 16 x a power of two take subnormal pivots, pivots above
2^1022 and infinite ones, as the reference's divisions do.

Rows of a diagonally dominant batch are scaled by powers of two (which changes no
solution), every fourth to where the pivot or its reciprocal is subnormal.  Bar: the tiled
path's 1e-12 relative to the serial Thomas of the same arrays; the scaled entries and
reciprocals keep 50 bits or more (2^-50 = 9e-16 a row)."""
import numpy as np
import pytest

from filtered_tdma_b200 import Solver
from filtered_tdma_b200 import _lib as L

pytestmark = pytest.mark.gpu

SHAPES = [(301, 100, False), (302, 250, False), (601, 700, False), (1001, 64, False),
          (300, 85, True), (301, 85, True), (603, 700, True), (600, 700, True), (301, 96, False)]


def batch(n_sys, n_row, seed, infinite):
    rng = np.random.default_rng(seed)
    A = -rng.uniform(0.2, 0.6, (n_row, n_sys))
    C = -rng.uniform(0.2, 0.6, (n_row, n_sys))
    B = rng.uniform(1.6, 1.9, (n_row, n_sys))
    D = rng.uniform(-0.9, 0.9, (n_row, n_sys))
    # pivots in [1.0, 1.9]: 2^1023 x pivot is finite and its reciprocal subnormal;
    # 2^-1023 x pivot is subnormal and its reciprocal finite
    e = rng.choice([0, 3, -2, 1023, -1023, 1022, -1022, 0], (n_row, n_sys))
    A, B, C, D = [np.ldexp(v, e) for v in (A, B, C, D)]
    if infinite:
        B[rng.uniform(size=B.shape) < 0.02] = np.inf
    return A, B, C, D


@pytest.mark.parametrize("n_sys,n_row,cyclic", SHAPES)
@pytest.mark.parametrize("infinite", [False, True])
def test_pivots_of_the_whole_range(cuda, orc, n_sys, n_row, cyclic, infinite):
    import torch
    arrays = batch(n_sys, n_row, n_sys + n_row, infinite)
    ref = orc.thomas_cyclic(*arrays) if cyclic else orc.thomas(*arrays)
    assert np.isfinite(ref).all()
    dev = [torch.from_numpy(np.ascontiguousarray(v)).to(cuda) for v in arrays]
    P = 5 if n_row < 256 else 16
    for flags in (L.FLAG_REFERENCE_ORDER, 0):
        s = Solver("pascal", n_sys, n_row, P, flags=flags)
        X = torch.empty_like(dev[3])
        s.solve_out(*dev, X, cyclic=cyclic)
        x = X.cpu().numpy()
        assert np.max(np.abs(x - ref)) <= 1e-12 * np.max(np.abs(ref)), flags
        assert s.status() == 0
