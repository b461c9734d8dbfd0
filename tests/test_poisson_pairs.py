"""The pair kernel of the Poisson solve at the edges of its range: one sub-segment, a
half-filled last warp, groups partly outside the modes, the longest columns, and
columns beyond it (the general kernel).  Bar as in test_poisson.py: the backward
error of every mode at most 1e-13 (the pinned mode's matrix is ill-conditioned)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1m,n2m,n3m", [(16, 6, 16), (34, 7, 48), (64, 64, 176), (30, 50, 400),
                                         (18, 16, 512), (18, 16, 544), (2, 1, 64),
                                         (190, 100, 96)])
def test_pairs_backward_error(cuda, n1m, n2m, n3m):
    import torch

    from filtered_tdma_b200.poisson import ChannelPoisson
    from oracle import poisson_oracle as O
    p = ChannelPoisson(n1m, n2m, n3m, gamma=1.5)
    rng = np.random.default_rng(n1m + n3m)
    rhs = rng.uniform(-1, 1, (n3m, p.n_modes)) + 1j * rng.uniform(-1, 1, (n3m, p.n_modes))
    hat = torch.from_numpy(rhs.copy()).to(cuda)
    p.solve(hat)
    x = hat.cpu().numpy()
    A, B, C = O.matrices(p.dz, p.dmz, p.lam, n3m)
    d = rhs.copy()
    d[0, 0] = 0.0
    r = d - B * x
    r[1:] -= A[1:] * x[:-1]
    r[:-1] -= C[:-1] * x[1:]
    scale = np.max(np.abs(A) + np.abs(B) + np.abs(C), axis=0) * np.max(np.abs(x), axis=0) + \
        np.max(np.abs(d), axis=0)
    assert np.max(np.max(np.abs(r), axis=0) / scale) <= 1e-13
    assert p.status() == 0
