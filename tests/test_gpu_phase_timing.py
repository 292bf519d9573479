"""Per-phase timing: its phases by name, and the same results with it on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PHASES = [(dict(pipeline=1, rng=1, exchange=1), ["mtgp32", "boxmuller", "sample_weight", "block_sort", "exchange", "resample"]),
          (dict(pipeline=1, rng=1, exchange=0, num_transfer=0), ["mtgp32", "boxmuller", "sample_weight", "block_sort", "resample"]),
          (dict(pipeline=1, rng=1, exchange=3),
           ["mtgp32", "boxmuller", "sample_weight", "block_sort", "a2a_merge", "exchange", "resample"]),
          (dict(pipeline=2, rng=1, exchange=1), ["mtgp32", "boxmuller", "sample_sort", "exchange_resample"]),
          (dict(pipeline=2, rng=0, exchange=2), ["sample_sort", "exchange_resample"]),
          (dict(pipeline=0, rng=0, exchange=1), ["step"])]


@pytest.mark.parametrize("kw,phases", PHASES)
def test_phases_by_name_and_the_same_results(gpu, kw, phases):
    """Timed and untimed filters in step, the timed one switched off half way."""
    E = gpu
    p = E.unicycle_params(2)
    inputs, _ = E.make_trace(0, p, 2, 8)
    cfg = dict(dict(particles_per_subfilter=128, num_subfilters=16, num_transfer=1, mtgp_streams=96), **kw)
    a, b = E.ParticleFilter(0, p, **cfg), E.ParticleFilter(0, p, **cfg)
    a.set_timing(True)
    for k in range(8):
        if k == 5:
            a.set_timing(False)
        x, y = a.step(inputs[k]), b.step(inputs[k])
        assert x.tobytes() == y.tobytes()
        if k < 5:
            t = a.last_step_timing()
            assert [n for n, _ in t] == phases and all(ms >= 0 for _, ms in t)
    assert np.array_equal(a.particles(), b.particles())
