"""Submitted steps at the queue's edges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNI = 0


def setup(E, steps):
    p = E.unicycle_params(6)
    inputs, _ = E.make_trace(UNI, p, 6, steps)
    return p, inputs, dict(particles_per_subfilter=256, num_subfilters=16, num_transfer=1, exchange=1)


def test_submit_is_refused_while_the_stream_is_captured(gpu):
    """A submit under capture is an error that leaves the filter as it was: nothing
    pending, and the steps after it those of a filter that never met it."""
    import torch
    E = gpu
    p, inputs, cfg = setup(E, 6)
    a, b = E.ParticleFilter(UNI, p, **cfg), E.ParticleFilter(UNI, p, **cfg)
    a.submit(inputs[0])
    got = list(a.collect())
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(torch.cuda.ExternalStream(a.stream())):
        g.capture_begin(capture_error_mode="thread_local")
        with pytest.raises(E.PFError) as ei:
            a.submit(inputs[1])
        g.capture_end()
    assert ei.value.status == E.PF_ERR_CUDA
    assert len(a.collect(wait=False)) == 0
    for k in range(1, 6):
        a.submit(inputs[k])
    got += list(a.collect())
    want = [b.step(inputs[k]) for k in range(6)]
    assert len(got) == 6
    assert all(x["mean"].tobytes() == y["mean"].tobytes() and x["step"] == y["step"] for x, y in zip(got, want))
    assert np.array_equal(a.particles(), b.particles())
