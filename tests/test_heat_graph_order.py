"""A graph step's first call for a field captures its graph without waiting for the
caller's queue and without running anything beside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_first_graph_step_does_not_wait(cuda):
    import torch

    from filtered_tdma_b200.heat import HeatADI
    h = HeatADI(48, 32, 64, dt=3e-4)
    a = h.field(cuda)
    b = a.clone()
    want = a.clone()
    h.step(want, 3, graph=False)
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    for th in (a, b):  # the first call, and the first for another field
        done = torch.cuda.Event()
        with torch.cuda.stream(st):
            torch.cuda._sleep(400_000_000)  # about 0.2 s, far above the capture's time
            h.step(th, 1, graph=False, stream=st.cuda_stream)
            done.record(st)
        h.step(th, 2, stream=st.cuda_stream)
        assert not done.query()  # the host came back while the sleep or step ran
        torch.cuda.synchronize()
        assert torch.equal(th, want)


def test_capture_beside_queued_steps(cuda):
    # eager steps of one field are still queued when another field's graph is captured
    import torch

    from filtered_tdma_b200.heat import HeatADI
    h = HeatADI(96, 128, 64, dt=3e-4)
    g = torch.Generator(device=cuda).manual_seed(3)
    start = torch.rand(h.shape, generator=g, device=cuda, dtype=torch.float64)
    want = start.clone()
    h.step(want, 21, graph=False)
    torch.cuda.synchronize()
    want = want.cpu().numpy()
    st = torch.cuda.Stream()
    for _ in range(5):
        a, b = start.clone(), start.clone()
        torch.cuda.synchronize()
        h.step(a, 20, graph=False, stream=st.cuda_stream)
        h.step(b, 21, stream=st.cuda_stream)
        h.step(a, 1, stream=st.cuda_stream)
        torch.cuda.synchronize()
        assert np.array_equal(a.cpu().numpy(), want)
        assert np.array_equal(b.cpu().numpy(), want)
