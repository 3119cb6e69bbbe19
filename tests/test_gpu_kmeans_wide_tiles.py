"""More than 64 clusters at the edges of the 64 x 16 tiles: ragged tiles, rows of
odd widths, tiles whose candidate list is longer than their 128 sums, negative
and large features (which leave the tile's 32-bit sums); labels equal the
FP32-exact oracle's and the centroids the FP64 means, within 1e-5 relative:
features are summed exactly after rounding to multiples of 2^-24."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,k,scale,shift", [
    (64, 16, 70, 1.0, 0.0), (65, 17, 70, 1.0, 0.0), (63, 33, 200, 1.0, 0.0),
    (130, 31, 300, 1.0, 0.0),              # noise: every cluster is a candidate
    (7, 50, 65, 1.0, -0.5), (96, 40, 100, 30000.0, 0.0), (1, 70, 65, 1.0, 0.0)])
@pytest.mark.parametrize("dim", [3, 5])
def test_tiles(cuda, w, h, k, scale, shift, dim):
    import torch
    from split_gb300 import kmeans
    rng = np.random.default_rng(w * h + dim)
    n = w * h
    feats = ((rng.random((dim, n)) + shift) * scale).astype(np.float32)
    c0 = feats[:, rng.choice(n, size=k, replace=n < k)].copy()
    cent = torch.from_numpy(c0).to(cuda)
    labels = torch.full((n,), -7, dtype=torch.int32, device=cuda)
    ws = kmeans.cluster(torch.from_numpy(feats).to(cuda), cent, labels, None, 1, -1.0, dim=dim,
                        width=w)
    torch.cuda.synchronize()
    ws.check("cluster")
    lab = labels.cpu().numpy()
    assert np.array_equal(lab, oracle.kmeans_assign_f32(feats, c0))
    want = oracle.kmeans_update_f64(lab, feats, c0)
    want = want[0] if isinstance(want, tuple) else want
    got = cent.cpu().numpy().astype(np.float64)
    assert (np.abs(got - want) <= 1e-5 * np.maximum(np.abs(want), 1e-3)).all()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e25])
@pytest.mark.parametrize("k", [64, 65, 128, 129, 1500])
@pytest.mark.parametrize("dim", [3, 5])
def test_no_distance_below_infinity(cuda, bad, k, dim):
    """Centroids from which every distance is infinite or NaN: all pixels carry
    label 0 and count in cluster 0, whatever sums their tile takes."""
    import torch
    from split_gb300 import kmeans
    w, h = 70, 45
    rng = np.random.default_rng(k + dim)
    feats = rng.random((dim, w * h)).astype(np.float32)
    c0 = np.full((dim, k), bad, dtype=np.float32)
    for one in (False, True):
        if one:   # and one finite centroid, which then gets every pixel
            c0[:, k // 2] = 0.5
        cent = torch.from_numpy(c0).to(cuda)
        labels = torch.full((w * h,), -7, dtype=torch.int32, device=cuda)
        ws = kmeans.cluster(torch.from_numpy(feats).to(cuda), cent, labels, None, 1, -1.0, dim=dim,
                            width=w)
        torch.cuda.synchronize()
        lab = labels.cpu().numpy()
        assert (lab == (k // 2 if one else 0)).all()
        got = cent.cpu().numpy()
        if k > 64:   # (the persistent kernel's update starts from the old centroid)
            ws.check("cluster")
            want = feats.astype(np.float64).mean(1)
            assert np.allclose(got[:, lab[0]], want, rtol=1e-5, atol=0)
        keep = np.arange(k) != lab[0]
        assert np.array_equal(got[:, keep], c0[:, keep], equal_nan=True)


@pytest.mark.parametrize("w,h,k", [
    (2000, 1, 70), (1, 2000, 70), (3000, 2, 200), (2, 3000, 200), (900, 5, 70), (5, 900, 1500),
    (33, 40, 70), (100, 9, 70), (1025, 1, 70),
    (64 * 32, 16, 70), (64 * 33, 16, 70),     # as many tiles as add directly, and one more
    (128, 64, 1500)])                         # two chunks of centroids in five dimensions
@pytest.mark.parametrize("layout", ["planar3", "planar5", "rgb3", "rgb5", "float5"])
def test_tile_shapes(cuda, w, h, k, layout):
    """Images whose rows or columns are shorter than a tile's, as flat as four
    pixels' runs and as noise, with features that depend on the place or not."""
    import torch
    from split_gb300 import kmeans
    rng = np.random.default_rng(w + h + k)
    n, dim = w * h, int(layout[-1])
    rgb = rng.integers(0, 256, (n, 3)).astype(np.uint8)
    rgb[n // 2:] = rgb[n // 2:n // 2 + 1]      # lanes and warps of one label
    c3 = (rgb.astype(np.float32) / np.float32(255)).T
    xy = np.stack([np.arange(n) % w, np.arange(n) // w]).astype(np.float32) * np.float32(0.02)
    feats = np.ascontiguousarray(np.concatenate([c3, xy])[:dim])
    c0 = feats[:, rng.choice(n, size=k, replace=n < k)].copy()
    if layout.startswith("planar"):
        pts, ly = torch.from_numpy(feats), kmeans.PLANAR
    elif layout.startswith("rgb"):
        pts, ly = torch.from_numpy(rgb), kmeans.RGB8
    else:
        pts, ly = torch.from_numpy(np.concatenate([c3.T, np.zeros((n, 1), np.float32)], 1)), \
            kmeans.FLOAT4
    cent = torch.from_numpy(c0).to(cuda)
    labels = torch.full((n,), -7, dtype=torch.int32, device=cuda)
    ws = kmeans.cluster(pts.contiguous().to(cuda), cent, labels, None, 1, -1.0, layout=ly, dim=dim,
                        width=w, xy_scale=0.02)
    ws.check("cluster")
    lab = labels.cpu().numpy()
    assert np.array_equal(lab, oracle.kmeans_assign_f32(feats, c0))
    want = oracle.kmeans_update_f64(lab, feats, c0)[0]
    got = cent.cpu().numpy().astype(np.float64)
    assert (np.abs(got - want) <= 1e-5 * np.maximum(np.abs(want), 1e-3)).all()
