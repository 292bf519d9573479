"""The step's faster routes at the sizes where they change: selection boundaries
that fall on integers, pairing rounds of the Vose build that take several
passes, estimates with one, four and sixteen warps per sub-filter, runs long
enough to replay graphs of several steps, the packed models against the scalar
ones, and the random buffer written in one launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UNICYCLE, DHARM, REFARM, BEACON, CAMARM = 0, 1, 2, 3, 4
BUILT = [(32, 1), (64, 2), (128, 2), (128, 4), (256, 2), (256, 4), (256, 8), (512, 2), (512, 4), (512, 16),
         (1024, 2), (1024, 4)]


@pytest.mark.parametrize("m,ppt", BUILT)
def test_systematic_boundaries_on_integers(gpu, O, m, ppt):
    """Cumulative sums that meet output positions exactly or within a rounding
    (equal and dyadic weights, uniforms at the ends of [0, 1)), and sums from
    1e-38 to 1e30: the oracle's selection, slot for slot."""
    base = np.stack([np.ones(m), 2.0 ** -(np.arange(m) % 8), np.where(np.arange(m) % 2, 1.0, 0.0),
                     np.where(np.arange(m) < 2, 1.0, 0.0)]).astype(np.float32)
    for u in (0.0, 2.0 ** -24, 0.5, 1.0 - 2.0 ** -24):
        for scale in (1.0, 1e-38, 1e30):
            w = (base * np.float32(scale)).astype(np.float32)
            us = np.full(len(w), u, np.float32)
            assert np.array_equal(gpu.resample(1, w.ravel(), us, m, ppt), O.resample(1, w.ravel(), us, m, ppt))


@pytest.mark.parametrize("m,ppt", BUILT)
def test_vose_rounds_of_many_pairs(gpu, O, m, ppt):
    """First rounds of m / 2 pairs (several passes over the CTA), of 33 and of 31
    pairs, and weights whose large entries stay large for many rounds."""
    rng = np.random.default_rng(m * 31 + ppt)
    w = np.full((5, m), 0.1, np.float32)
    w[0, ::2] = 1.9
    w[1, :min(33, m // 2)] = 3.0
    w[2, :min(31, m // 2)] = 5.0
    w[3] = rng.exponential(1, m)
    w[4] = rng.exponential(1, m) ** 6
    u = rng.random(10 * m).astype(np.float32)
    assert np.array_equal(gpu.resample(2, w.ravel(), u, m, ppt), O.resample(2, w.ravel(), u, m, ppt))


@pytest.mark.parametrize("S,angles", [(1, 0), (3, 1), (4, 4), (5, 2), (16, 16)])
@pytest.mark.parametrize("m,nsub,shift", [(1, 7, 0), (100, 5, 0), (777, 3, 0), (32, 296, 0), (32, 297, 1), (250, 1184, 0),
                                          (64, 1185, 0), (512, 2048, 0), (1028, 300, 0), (5000, 4, 0)])
def test_estimate_of_given_particles(gpu, S, angles, m, nsub, shift):
    """Against FP64 sums of the same keys.  The FP32 weights are within
    (2 + |k - max|) 2^-22 of the exponential (keys span 30), so each mean is
    within 2 * 32 * 2^-22 of the FP64 one relative to the largest value, and a
    circular mean within that over its resultant length (above 0.9 here).
    shift: the arrays start one float past a 16-byte boundary."""
    import torch
    E = gpu
    rng = np.random.default_rng(S * 1000 + m)
    T = m * nsub
    keys = -30.0 * rng.random(T).astype(np.float32)
    x = rng.normal(0.5, 0.2, (S, T)).astype(np.float32)
    dk = torch.zeros(T + 4, device="cuda")
    ds = torch.zeros(S * T + 4, device="cuda")
    dk[shift:shift + T] = torch.from_numpy(keys).cuda()
    ds[shift:shift + S * T] = torch.from_numpy(x.ravel()).cuda()
    out = torch.zeros(E.ESTIMATE_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    mask = ((1 << angles) - 1) << (S - angles)
    for _ in range(2):  # the second call finds the ticket and the scratch as the first left them
        torch.cuda.synchronize()
        E.estimate_noalloc(dk.data_ptr() + 4 * shift, ds.data_ptr() + 4 * shift, S, T, m, out.data_ptr(), mask, 1)
        torch.cuda.synchronize()
        e = out.cpu().numpy().view(E.ESTIMATE_DTYPE)[0]
        k = keys.astype(np.float64)
        w = np.exp(k - k.max())
        tol = 2 * 32 * 2.0 ** -22
        for v in range(S):
            xv = x[v].astype(np.float64)
            if v >= S - angles:
                ref = np.arctan2((w * np.sin(xv)).sum(), (w * np.cos(xv)).sum())
                assert abs(e["mean"][v] - ref) <= tol / 0.9 + 1e-6  # __sincosf: 2^-21 absolute
            else:
                assert abs(e["mean"][v] - (w * xv).sum() / w.sum()) <= tol * np.abs(xv).max()
        assert abs(e["log_norm"] - (k.max() + np.log(w.sum()))) <= tol
        best = int(np.argmax(keys))
        assert e["best_subfilter"] == best // m and e["best_key"] == keys[best] and e["flags"] == 0
        assert np.array_equal(e["best"][:S], x[:, best])


def test_estimate_with_a_sub_filter_of_nan_keys(gpu):
    """NaN keys win nothing and are reported, whichever sub-filter holds them."""
    keys = np.full(4 * 64, -1.0, np.float32)
    keys[70] = -0.5
    keys[128:192] = np.nan
    e = gpu.estimate(keys, np.zeros((2, 256), np.float32), 64)
    assert e["flags"] == 1 and e["best_subfilter"] == 1 and e["best_key"] == np.float32(-0.5)


@pytest.mark.parametrize("model,pipe,kw", [
    (UNICYCLE, 2, {}), (UNICYCLE, 2, dict(exchange_period=3)), (UNICYCLE, 2, dict(exchange=3)),
    (UNICYCLE, 2, dict(num_subfilters=1, exchange=0, num_transfer=0)), (UNICYCLE, 2, dict(ess_fraction=0.5)),
    (UNICYCLE, 2, dict(resampler=2)), (UNICYCLE, 2, dict(resampler=0, resampling_freq=0.7)),
    (UNICYCLE, 2, dict(rng=1)), (UNICYCLE, 0, {}), (DHARM, 2, {}), (REFARM, 1, dict(rng=1, resampler=0, log_weights=0)),
    (UNICYCLE, 2, dict(num_subfilters=2048, particles_per_subfilter=128))])
def test_long_run_equals_steps(gpu, model, pipe, kw):
    """70 + 16 + 7 steps over device arrays (graphs of 16, 4 and 1 steps, the
    input ring wrapping) against pf_step: every estimate and the particles."""
    import torch
    E = gpu
    p = {UNICYCLE: lambda: E.unicycle_params(4), DHARM: lambda: E.dharm_params(4), REFARM: E.refarm_params}[model]()
    cap, parts = 40, (70, 16, 7)
    if model == REFARM:
        rng = np.random.default_rng(4)
        inputs = np.zeros(cap, E.STEP_INPUT_DTYPE)
        inputs["control"][:, :5] = rng.normal(0, 0.05, (cap, 5))
        inputs["meas"][:, :5] = 2.3 + rng.normal(0, 0.1, (cap, 5))
        inputs["meas"][:, 5:7] = rng.normal(0, 1, (cap, 2))
    else:
        inputs, _ = E.make_trace(model, p, 4, cap)
    cfg = dict(dict(particles_per_subfilter=256, num_subfilters=40, num_transfer=2, exchange=1, pipeline=pipe), **kw)
    a, b = E.ParticleFilter(model, p, **cfg), E.ParticleFilter(model, p, **cfg)
    din = torch.from_numpy(inputs.view(np.uint8).reshape(-1).copy()).cuda()
    n = sum(parts)
    dest = torch.zeros(cap * E.ESTIMATE_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    got = []
    a.run_device(din.data_ptr(), dest.data_ptr(), cap, parts[0])
    for k in parts[1:]:
        a.run_continue(k)
    a.synchronize()
    got = dest.cpu().numpy().view(E.ESTIMATE_DTYPE)
    ref = [b.step(inputs[k % cap]) for k in range(n)]
    for k in range(n - cap, n):
        assert got[k % cap].tobytes() == ref[k].tobytes(), k
    assert np.array_equal(a.particles(), b.particles())


@pytest.mark.parametrize("model,m,ppt", [(UNICYCLE, 512, 16), (UNICYCLE, 256, 8), (UNICYCLE, 128, 2), (UNICYCLE, 32, 1),
                                         (DHARM, 256, 2), (DHARM, 128, 4), (DHARM, 32, 1), (BEACON, 512, 16),
                                         (BEACON, 256, 2), (BEACON, 32, 1), (REFARM, 256, 2), (CAMARM, 256, 4)])
def test_packed_models_equal_scalar_models(gpu, model, m, ppt):
    """One step of the split pipeline (two particles to an instruction) on the
    reference layout's random numbers, against the scalar model on the same
    numbers: sorted keys and particles bit for bit; the random numbers are a
    single stream's of several generation chunks, from the separate generator
    and Box-Muller entry points."""
    E = gpu
    S, K, _, _ = E.model_info(model)
    p = {UNICYCLE: lambda: E.unicycle_params(7, 5), DHARM: lambda: E.dharm_params(7), BEACON: E.beacon_params,
         REFARM: E.refarm_params, CAMARM: E.camarm_params}[model]()
    N = 12
    T = N * m
    rng = np.random.default_rng(m + model)
    inp = np.zeros(1, E.STEP_INPUT_DTYPE)[0]
    inp["control"][:5] = rng.normal(0.3, 0.2, 5)
    inp["meas"] = rng.normal(2.0, 1.0, 16)
    start = np.tile(np.array(p.init_state[:S], np.float32)[:, None], (1, T)) + rng.normal(0, 0.3, (S, T)).astype(np.float32)
    per = -(-(K * T + (m + 1) * N) // 768) * 768
    words = E.mtgp_generate(1, 99, per, kind=1).view(np.float32)
    noise = E.boxmuller(words[:2 * ((K * T + 1) // 2)])[:K * T].reshape(K, T)
    state, ll = E.model_step(model, p, inp, start, noise)
    f = E.ParticleFilter(model, p, particles_per_subfilter=m, particles_per_thread=ppt, num_subfilters=N,
                         num_transfer=0, exchange=0, pipeline=E.PIPELINE_SPLIT, rng=E.RNG_REFLAYOUT, mtgp_streams=1,
                         seed=99)
    f.set_particles(start)
    f.step(inp)
    rows, keys = f.sorted()
    # the network's own permutation: particles whose keys tie keep its order
    want, idx = E.bitonic_sort(ll, m)
    order = (idx.reshape(N, m) + m * np.arange(N)[:, None]).ravel()
    assert np.array_equal(keys, want)
    assert np.array_equal(rows, state[:, order])
