"""The shared-matrix sweeps (two systems a thread) at the edges of their ranges: one
sub-segment, counts that leave the last warp half filled, the longest, and axes
beyond them (the general kernels), against the oracle.

Bars as in test_heat.py / test_momentum.py: 1e-12 relative to the largest value.
Grids 176, 240 and 288 long in x or y came out wrong before these sweeps (a copy
loop of half-filled warps left rows out).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ix,iy,iz", [
    (16, 16, 16), (48, 80, 48), (176, 32, 32), (32, 240, 16), (16, 288, 32), (304, 16, 16),
    (320, 32, 16), (16, 16, 512), (512, 16, 16), (16, 512, 16), (80, 48, 400),
    (16, 16, 544), (544, 16, 16), (16, 544, 16)])
def test_heat_grids(cuda, ix, iy, iz):
    import torch

    from filtered_tdma_b200.heat import HeatADI
    from oracle import heat_oracle as H
    dt = 3e-4
    th = H.initial(ix, iy, iz) + 0.1 * np.random.default_rng(ix + iy).uniform(
        -1, 1, (iz + 2, iy + 2, ix + 2))
    ref = H.step(H.step(th, dt), dt)
    h = HeatADI(ix, iy, iz, dt=dt)
    dev = torch.from_numpy(th).to(cuda)
    h.step(dev, 1, graph=False)
    h.step(dev, 1)
    got = dev.cpu().numpy()
    c = (slice(1, -1),) * 3
    assert np.max(np.abs(got[c] - ref[c])) <= 1e-12 * np.max(np.abs(ref[c]))
    assert np.array_equal(got[0], th[0]) and np.array_equal(got[:, :, 0], th[:, :, 0])


@pytest.mark.parametrize("nx,ny,nz", [(16, 16, 16), (32, 64, 48), (64, 32, 176), (16, 512, 16),
                                      (512, 16, 32), (16, 16, 512), (16, 16, 544),
                                      (1024, 16, 16)])
@pytest.mark.parametrize("comp", [0, 2])
def test_momentum_grids(cuda, nx, ny, nz, comp):
    import torch

    from filtered_tdma_b200.momentum import ChannelMomentum
    from oracle import momentum_oracle as O
    rng = np.random.default_rng(nx + nz + comp)
    rhs = rng.uniform(-1, 1, (nz + 2, ny + 2, nx + 2))
    m = ChannelMomentum(nx, ny, nz)
    ref = O.adi(rhs, m.metrics, comp, 1e-3, m.pbc)
    dev = torch.from_numpy(rhs).to(cuda)
    q = torch.full_like(dev, 5.0)
    m.adi(comp, dev, q, 1e-3)
    got = q.cpu().numpy()
    c = (slice(1, -1),) * 3
    assert np.max(np.abs(got[c] - ref[c])) <= 1e-12 * np.max(np.abs(ref[c]))
    assert (got[0] == 5.0).all() and (got[:, 0] == 5.0).all() and (got[:, :, -1] == 5.0).all()
    assert m.status() == 0
