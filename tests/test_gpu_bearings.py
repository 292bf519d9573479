"""Bearings at the ends of atan2's range: a landmark's offset that is zero or
subnormal, and a bearing measurement that is not a number -- through the scalar
model, the packed one and two threads per particle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNICYCLE = 0


def still(E, landmarks=1):
    """A unicycle that stays where it is, landmark 0 at the origin."""
    p = E.unicycle_params(1, landmarks)
    for i in range(3):
        p.sigma_q[i] = 0.0
    p.landmarks[0][0] = p.landmarks[0][1] = 0.0
    return p


def offsets(n):
    """n offsets whose length runs from 2^-100 to the smallest subnormal, some of them zero."""
    k = np.arange(n)
    a = 2 * np.pi * ((k * 0.381966) % 1.0)
    x = np.stack([np.cos(a), np.sin(a)]) * 2.0 ** -(100.0 + 50.0 * k / n)
    x[:, ::17] = 0.0
    return x.astype(np.float32)


def test_bearing_of_tiny_offsets(gpu):
    """The scalar model against FP64 atan2 of the same offsets.  The range is 0
    (its square underflows), so the log-likelihood is -(bearing / sigma)^2 / 2:
    within 3e-7 of the bearing from atan2, 2^-21 relative from the quotient's
    three roundings and the squares'."""
    E = gpu
    p = still(E)
    n = 512
    x = offsets(n)
    inp = np.zeros(1, E.STEP_INPUT_DTYPE)[0]
    _, ll = E.model_step(UNICYCLE, p, inp, np.concatenate([-x, np.zeros((1, n), np.float32)]), np.zeros((3, n), np.float32))
    ref = np.arctan2(x[1].astype(np.float64), x[0].astype(np.float64))
    got = np.sqrt(-2.0 * ll.astype(np.float64)) * np.float64(np.float32(p.sigma_bearing))
    assert np.all(np.abs(got - np.abs(ref)) <= 3e-7 + 2.0 ** -21 * np.abs(ref))


@pytest.mark.parametrize("m,ppt,tpp,pipe", [(256, 4, 1, 2), (256, 2, 1, 2), (512, 16, 1, 2), (32, 1, 1, 2),
                                            (256, 4, 1, 0), (256, 2, 2, 2)])
@pytest.mark.parametrize("nan", [False, True])
def test_keys_at_a_landmark(gpu, m, ppt, tpp, pipe, nan):
    """Particles on and beside a landmark, with and without a bearing that is not
    a number among the measurements: the filter's keys are the scalar model's (two
    threads per particle add the six squares in another order: 2^-21)."""
    E = gpu
    N = 4
    p = still(E, 3)
    inp = np.zeros(1, E.STEP_INPUT_DTYPE)[0]
    inp["meas"][:3] = 1.0, 2.0, 3.0
    inp["meas"][3:6] = 0.3, np.nan if nan else -0.4, 0.5
    T = N * m
    x = np.zeros((3, T), np.float32)
    x[:2] = -offsets(T)
    x[:2, ::3] = np.random.default_rng(3).normal(0, 2, (2, len(range(0, T, 3)))).astype(np.float32)
    _, ll = E.model_step(UNICYCLE, p, inp, x, np.zeros((3, T), np.float32))
    assert np.all(np.isfinite(ll))
    f = E.ParticleFilter(UNICYCLE, p, particles_per_subfilter=m, particles_per_thread=ppt, threads_per_particle=tpp,
                         num_subfilters=N, num_transfer=0, exchange=0, pipeline=pipe)
    f.set_particles(x)
    e = f.step(inp)
    _, keys = f.sorted()
    want = -np.sort(-ll.reshape(N, m), axis=1)
    keys = keys.reshape(N, m)
    assert np.array_equal(keys, want) if tpp == 1 else np.all(np.abs(keys - want) <= 2.0 ** -21 * np.abs(want))
    assert e["flags"] == 0 and np.all(np.isfinite(e["mean"][:3]))


def test_bearing_that_is_not_a_number_says_nothing(gpu):
    """The log-likelihood with a NaN bearing is that of the other measurements:
    the whole one less the landmark's bearing term, which a bearing measured
    where the particle sees the landmark makes 0 up to (6e-7 / sigma)^2 / 2 and
    the roundings of sums below 2^10 (2^-13)."""
    E = gpu
    p = still(E, 3)
    n = 64
    x = np.concatenate([np.random.default_rng(5).normal(0, 2, (2, n)), np.zeros((1, n))]).astype(np.float32)
    inp = np.zeros(1, E.STEP_INPUT_DTYPE)[0]
    inp["meas"][:3] = 1.0, 2.0, 3.0
    inp["meas"][3:6] = 0.3, np.nan, 0.5
    _, ll = E.model_step(UNICYCLE, p, inp, x, np.zeros((3, n), np.float32))
    for i in range(n):
        seen = inp.copy()
        seen["meas"][4] = np.arctan2(np.float64(p.landmarks[1][1]) - x[1, i], np.float64(p.landmarks[1][0]) - x[0, i])
        _, one = E.model_step(UNICYCLE, p, seen, x[:, i:i + 1], np.zeros((3, 1), np.float32))
        assert abs(ll[i] - one[0]) <= 0.5 * (6e-7 / p.sigma_bearing) ** 2 + 2.0 ** -13 * max(1.0, abs(one[0]) / 1024)
