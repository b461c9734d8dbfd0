"""The heat step on fields at every 8-byte offset of a 32-byte line: the fused Z sweep
reads 16-byte aligned fields, the others take the right-hand side as a pass of its own,
and the X sweep's stores follow the offset.  Bar as in test_heat.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ix,iy,iz", [(48, 32, 16), (16, 16, 16), (48, 80, 48), (32, 32, 272)])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
def test_unaligned_fields(cuda, ix, iy, iz, offset):
    import torch

    from filtered_tdma_b200.heat import HeatADI
    from oracle import heat_oracle as H
    dt = 3e-4
    th = H.initial(ix, iy, iz) + 0.1 * np.random.default_rng(ix + iz).uniform(
        -1, 1, (iz + 2, iy + 2, ix + 2))
    ref = H.step(H.step(th, dt), dt)
    flat = torch.full((th.size + 4,), 7.0, dtype=torch.float64, device=cuda)
    dev = flat[offset:offset + th.size].view(th.shape)
    dev.copy_(torch.from_numpy(th))
    h = HeatADI(ix, iy, iz, dt=dt)
    h.step(dev, 1)
    h.step(dev, 1, graph=False)
    got = dev.cpu().numpy()
    c = (slice(1, -1),) * 3
    assert np.max(np.abs(got[c] - ref[c])) <= 1e-12 * np.max(np.abs(ref[c]))
    assert np.array_equal(got[0], th[0]) and np.array_equal(got[:, :, 0], th[:, :, 0])
    assert (flat[:offset] == 7.0).all() and (flat[offset + th.size:] == 7.0).all()
