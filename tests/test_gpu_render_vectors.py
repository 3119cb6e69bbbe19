"""Label ranks, segment means and painting, four pixels per thread: sizes that
end inside a vector, a warp or a scan tile, labels and outputs that start off a
16-byte boundary, segments without members, features inside and outside [0, 1]
in one warp.  Ranks equal the oracle's; means are the FP64 quotients of exact
integer sums, rounded once; painted values are the means'."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _at(values, offset, device):
    """A device copy that starts `offset` elements past a 16-byte boundary."""
    import torch
    t = torch.from_numpy(np.ascontiguousarray(values))
    buf = torch.empty(t.numel() + 4, dtype=t.dtype, device=device)
    view = buf[offset:offset + t.numel()].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("n,offset", [
    (1, 0), (3, 1), (4, 0), (127, 0), (128, 2), (1023, 3), (1024, 0), (4097, 0),
    (131071, 0), (131072, 1), (262145, 0)])     # 4096 words of the scan hold 131071 labels and -1
def test_ranks(cuda, n, offset):
    from split_gb300 import ccl
    rng = np.random.default_rng(n)
    runs = np.repeat(rng.integers(-1, n, size=n), rng.integers(1, 9, size=n))[:n].astype(np.int32)
    for lab in (runs, np.arange(n, dtype=np.int32), np.full(n, -1, np.int32),
                np.full(n, n - 1, np.int32)):
        want, count = oracle.compress_labels(lab)
        got = _at(lab, offset, cuda)
        assert ccl.compress_labels(got) == count
        assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("n,offset,k", [(1, 0, 65), (130, 1, 70), (4096, 0, 300), (4098, 2, 300),
                                        (33333, 0, 5000), (65536, 0, 100)])
@pytest.mark.parametrize("wide", [False, True])
def test_means_and_paint(cuda, n, offset, k, wide):
    import torch
    from split_gb300 import kmeans
    rng = np.random.default_rng(n + k)
    lab = np.repeat(rng.integers(-2, k + 1, size=n), rng.integers(1, 40, size=n))[:n]
    lab = lab.astype(np.int32)
    pts = rng.random((3, n), dtype=np.float32)
    pts[:, ::7] = 1.0
    pts[:, 1::11] = 0.0
    if wide:      # some warps hold values outside [0, 1]
        far = rng.random(n) < 0.004
        far[0] = True
        pts[:, far] = (rng.random((3, far.sum())) * 2000 - 1000).astype(np.float32)
    old = rng.random((3, k), dtype=np.float32)
    q = np.rint(pts.astype(np.float64) * 2.0**24).astype(np.int64)
    inside = (lab >= 0) & (lab < k)
    want = old.copy()
    count = np.bincount(lab[inside], minlength=k)
    for d in range(3):
        s = np.zeros(k, np.int64)
        np.add.at(s, lab[inside], q[d, inside])
        has = count > 0
        want[d, has] = (s[has].astype(np.float64) / 2.0**24 / count[has]).astype(np.float32)
    dev_lab, cent = _at(lab, offset, cuda), torch.from_numpy(old).to(cuda)
    kmeans.calculate_centroids(dev_lab, _at(pts, offset, cuda), cent)
    assert np.array_equal(cent.cpu().numpy(), want)
    out = _at(np.full((3, n), -5.0, np.float32), offset, cuda)
    kmeans.propagate_centroids(dev_lab, cent, out)
    assert np.array_equal(out.cpu().numpy(),
                          np.where(inside, want[:, np.where(inside, lab, 0)], np.float32(0)))


@pytest.mark.parametrize("scale", [100.0, -1e6, 1e10, 2.0e11])
@pytest.mark.parametrize("n,offset", [(5, 0), (127, 1), (4096, 0), (4098, 2), (33333, 3)])
def test_means_of_large_features(cuda, n, offset, scale):
    """Features outside [0, 1] everywhere: 64-bit sums of runs below 2^32, 96-bit
    words above, in runs shorter and longer than a thread's four pixels."""
    import torch
    from split_gb300 import kmeans
    k = 70
    rng = np.random.default_rng(n)
    lab = np.repeat(rng.integers(-1, k + 1, size=n), rng.integers(1, 9, size=n))[:n].astype(np.int32)
    pts = ((rng.random((3, n)) - 0.25) * scale).astype(np.float32)
    q = np.rint(pts.astype(np.float64) * 2.0**24).astype(np.int64)   # exact: floats have 24 bits
    inside = (lab >= 0) & (lab < k)
    old = rng.random((3, k), dtype=np.float32)
    want = old.copy()
    for c in np.unique(lab[inside]):
        for d in range(3):
            total = sum(int(v) for v in q[d, lab == c])
            want[d, c] = np.float32(float(total) / 2.0**24 / int((lab == c).sum()))
    cent = torch.from_numpy(old).to(cuda)
    ws = kmeans.calculate_centroids(_at(lab, offset, cuda), _at(pts, offset, cuda), cent)
    ws.check("calculate_centroids")
    assert np.array_equal(cent.cpu().numpy(), want)
