"""Estimates of given particles whose sub-filters are longer than what a team of
warps holds in registers (the rest is read in loops), one to sixteen warps a
sub-filter, rows that are and are not 16-byte aligned, log and linear weights."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,angles", [(3, 1), (6, 2)])
@pytest.mark.parametrize("m,nsub,shift,linear", [
    (1024, 1185, 0, 0), (1024, 1185, 0, 1), (777, 1200, 0, 0), (250, 1185, 0, 0), (512, 2048, 1, 0), (512, 2048, 1, 1),
    (2500, 300, 0, 0), (1030, 300, 0, 0), (1030, 300, 0, 1), (9000, 3, 0, 0), (4500, 3, 1, 0), (4500, 3, 1, 1)])
def test_estimate_of_long_sub_filters(gpu, S, angles, m, nsub, shift, linear):
    """Against FP64 sums of the same keys.  Log weights: the FP32 weights are
    within (2 + |k - max|) 2^-22 of the exponential (keys span 30), so a mean is
    within 2 * 32 * 2^-22 of the FP64 one relative to the largest value, and a
    circular mean within that over its resultant length (above 0.9 here) and
    __sincosf's 2^-21.  Linear weights are used as they are: 1e-11, the FP64
    sums' roundings."""
    import torch
    E = gpu
    rng = np.random.default_rng(S * 1000 + m)
    T = m * nsub
    keys = -30.0 * rng.random(T).astype(np.float32)
    if linear:
        keys = np.exp(keys)
    x = rng.normal(0.5, 0.2, (S, T)).astype(np.float32)
    dk = torch.zeros(T + 4, device="cuda")
    ds = torch.zeros(S * T + 4, device="cuda")
    dk[shift:shift + T] = torch.from_numpy(keys).cuda()
    ds[shift:shift + S * T] = torch.from_numpy(x.ravel()).cuda()
    out = torch.zeros(E.ESTIMATE_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    E.estimate_noalloc(dk.data_ptr() + 4 * shift, ds.data_ptr() + 4 * shift, S, T, m, out.data_ptr(),
                       ((1 << angles) - 1) << (S - angles), 1 - linear)
    torch.cuda.synchronize()
    e = out.cpu().numpy().view(E.ESTIMATE_DTYPE)[0]
    k = keys.astype(np.float64)
    top = 0.0 if linear else k.max()
    w = k if linear else np.exp(k - top)
    tol = 1e-11 if linear else 2 * 32 * 2.0 ** -22
    for v in range(S):
        xv = x[v].astype(np.float64)
        if v >= S - angles:
            ref = np.arctan2((w * np.sin(xv)).sum(), (w * np.cos(xv)).sum())
            assert abs(e["mean"][v] - ref) <= tol / 0.9 + 1e-6
        else:
            assert abs(e["mean"][v] - (w * xv).sum() / w.sum()) <= tol * np.abs(xv).max()
    assert abs(e["log_norm"] - (top + np.log(w.sum()))) <= tol * max(1.0, abs(e["log_norm"]))
    best = int(np.argmax(keys))
    assert e["best_subfilter"] == best // m and e["best_key"] == keys[best] and e["flags"] == 0
    assert np.array_equal(e["best"][:S], x[:, best])
