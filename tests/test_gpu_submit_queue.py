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


YIELD_CHILD = r"""
import ctypes, sys
cu = ctypes.CDLL("libcuda.so.1")
assert cu.cuInit(0) == 0
flags = int(sys.argv[1])
assert cu.cuDevicePrimaryCtxSetFlags_v2(0, flags) == 0
sys.path.insert(0, sys.argv[2])
import numpy as np
import esthera_b200 as E
count = ctypes.CDLL(sys.argv[3]).yields
p = E.unicycle_params(6)
inputs, _ = E.make_trace(0, p, 6, 32)
f = E.ParticleFilter(0, p, particles_per_subfilter=512, num_subfilters=4096, num_transfer=1, exchange=1)
f.submit(inputs[0])
f.collect()
for k in range(1, 32):
    f.submit(inputs[k])
n = count()
got = f.collect()
print(len(got), int(got[-1]["step"]), count() - n)
"""


@pytest.mark.parametrize("flag,yields", [(0x1, False), (0x2, True)])
def test_collect_follows_the_schedule_flag(gpu, tmp_path, flag, yields):
    """A waiting collect gives its core away on a device set to yield
    (CU_CTX_SCHED_YIELD), and not on one set to spin: sched_yield counted by a
    preloaded library, in a process of its own."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    src, lib = tmp_path / "yields.c", tmp_path / "yields.so"
    src.write_text("static long n; int sched_yield(void) { __atomic_fetch_add(&n, 1, __ATOMIC_RELAXED); return 0; }\n"
                   "long yields(void) { return __atomic_load_n(&n, __ATOMIC_RELAXED); }\n")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(lib), str(src)], check=True)
    r = subprocess.run([sys.executable, "-c", YIELD_CHILD, str(flag), str(Path(gpu.__file__).parents[1]), str(lib)],
                       env=dict(os.environ, LD_PRELOAD=str(lib), OPENBLAS_NUM_THREADS="1"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    n, step, seen = map(int, r.stdout.split())
    assert (n, step) == (31, 32)
    assert (seen > 0) == yields
