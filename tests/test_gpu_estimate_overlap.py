"""Estimates of given particles that run beside one another: pfk_estimate owns
its scratch, so it and replays of a captured pfk_estimate_noalloc may overlap in
any way, and neither may leave anything behind for later calls."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def particles(seed, m, n):
    rng = np.random.default_rng(seed)
    return (-30.0 * rng.random(m * n)).astype(np.float32), rng.normal(0.5, 0.2, (3, m * n)).astype(np.float32)


def same(a, b):
    return all(np.array_equal(a[f], b[f]) for f in ("mean", "log_norm", "best", "best_key", "best_subfilter", "flags"))


def test_estimate_beside_replays_of_the_allocation_free_one(gpu):
    import torch
    E = gpu
    m, n = 512, 2048
    keys, x = particles(1, m, n)
    dk, dx = torch.from_numpy(keys).cuda(), torch.from_numpy(x).cuda()
    out = torch.zeros(E.ESTIMATE_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    s = torch.cuda.Stream(priority=-1)  # replays start while the other call's CTAs are still to come
    torch.cuda.synchronize()

    def call(stream):
        E.estimate_noalloc(dk.data_ptr(), dx.data_ptr(), 3, m * n, m, out.data_ptr(), 4, 1, stream)

    call(s.cuda_stream)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        call(s.cuda_stream)

    # many small sub-filters: thousands of CTAs that end one after the other, so
    # that replays run beside each call
    sets = [particles(seed, 4, 60000) for seed in (2, 3)]
    alone = [E.estimate(k, v[:1], 4) for k, v in sets]
    wrong, done = [], threading.Event()

    def other():
        try:
            for i in range(1600):
                k, v = sets[i % 2]
                if not same(E.estimate(k, v[:1], 4), alone[i % 2]):
                    wrong.append(i)
        finally:
            done.set()

    t = threading.Thread(target=other)
    t.start()
    with torch.cuda.stream(s):
        while not done.is_set():
            for _ in range(16):
                g.replay()
            s.synchronize()
    t.join()
    assert not wrong
    # and afterwards, alone, over other particles in turn: replays of the captured
    # call, then more plain calls than it keeps anything for
    fresh = [particles(seed, m, n) for seed in (4, 5)]
    ref = [E.estimate(k, v, m, 4) for k, v in fresh]
    for i in range(400):
        k, v = fresh[i % 2]
        dk.copy_(torch.from_numpy(k))
        dx.copy_(torch.from_numpy(v))
        out.zero_()
        torch.cuda.synchronize()
        if i < 100:
            g.replay()
        else:
            call(s.cuda_stream)
        torch.cuda.synchronize()
        assert same(out.cpu().numpy().view(E.ESTIMATE_DTYPE)[0], ref[i % 2]), i
    assert same(E.estimate(sets[0][0], sets[0][1][:1], 4), alone[0])
