"""Clustering straight from the image bytes, in pipelines and batches: equal bit
for bit to kmeans.cluster on the packed float4 features, at sizes that end
inside a span (64 x 16), a batch of rows (4) or a pixel vector (4), at bytes off
a word boundary, for three dimensions (two batches of rows per step) and five;
batches of more images than blocks; and the pipeline
without erosion, whose one relabel writes the merged segments."""
import numpy as np
import pytest

import oracle
from split_gb300 import synth

pytestmark = pytest.mark.gpu


def _t(a, dev):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def _centroids(seed, rgb, k, dim):
    """k pixels' features, a pixel possibly more than once (few pixels)."""
    f = synth.features(rgb, dim)
    return f[:, np.random.default_rng(seed).integers(0, f.shape[1], size=k)]


@pytest.mark.parametrize("w,h,offset", [
    (64, 16, 0), (64, 17, 0), (65, 15, 0), (63, 33, 1), (128, 7, 0), (200, 130, 3),
    (257, 96, 2), (1, 90, 0), (90, 1, 1), (5, 3, 0), (640, 203, 0)])
@pytest.mark.parametrize("dim,k,threshold", [(3, 8, -1.0), (5, 16, -1.0), (3, 33, 0.001)])
def test_pipeline_bytes_equal_float4(cuda, w, h, offset, dim, k, threshold):
    import torch
    from split_gb300 import kmeans, pipeline
    rgb = synth.voronoi_rgb8(7 * w + h, w, h, 12, sigma=8.0)
    c0 = _centroids(7 * w + h, rgb, k, dim)
    buf = torch.empty(rgb.size + 4, dtype=torch.uint8, device=cuda)
    dev = buf[offset:offset + rgb.size].view(h, w, 3)
    dev.copy_(torch.from_numpy(rgb))
    pipe = pipeline.Pipeline(w, h, pipeline.Params(
        nclusters=k, dim=dim, kmeans_iters=9, kmeans_threshold=threshold, merge_P=8,
        compute_normals=False), cuda)
    pipe.run(dev, _t(c0, cuda))
    f4 = np.zeros((w * h, 4), np.float32)
    f4[:, :3] = synth.features(rgb, 3).T
    cent, labels = _t(c0, cuda), torch.empty(w * h, dtype=torch.int32, device=cuda)
    ws = kmeans.cluster(_t(f4, cuda), cent, labels, None, 9, threshold,
                        layout=kmeans.FLOAT4 | kmeans.UNIT_RANGE, dim=dim, width=w)
    torch.cuda.synchronize()
    pipe.ws.check("pipeline")
    ws.check("cluster")
    assert torch.equal(pipe.cluster_labels, labels)
    assert torch.equal(pipe.centroids, cent)


@pytest.mark.parametrize("dim,threshold", [(5, -1.0), (3, 0.002)])
def test_batch_of_many_small_images(cuda, dim, threshold):
    """700 images of 1 to 4000 pixels and one larger: a block's part of the work
    covers several whole images."""
    import torch
    from split_gb300 import batch, pipeline
    rng = np.random.default_rng(dim)
    shapes = [(int(rng.integers(1, 9)) if i % 3 else int(rng.integers(1, 64)),
               int(rng.integers(1, 9)) if i % 3 else int(rng.integers(1, 64)),
               int(rng.integers(1, 6)), int(rng.integers(1, 7))) for i in range(700)]
    shapes.insert(77, (700, 400, 16, 8))
    params = pipeline.Params(dim=dim, merge_P=8, kmeans_threshold=threshold)
    imgs = [synth.voronoi_rgb8(i, w, h, 4, sigma=4.0) for i, (w, h, _, _) in enumerate(shapes)]
    cents = [_centroids(i, imgs[i], k, dim) for i, (_, _, k, _) in enumerate(shapes)]
    b = batch.Batch(shapes, params, cuda)
    b.load(imgs, cents)
    b.run()
    torch.cuda.synchronize()
    for i, (w, h, k, iters) in enumerate(shapes):
        p = pipeline.Params(**{**params.__dict__, "nclusters": k, "kmeans_iters": iters})
        one = pipeline.Pipeline(w, h, p, cuda)
        one.run(_t(imgs[i], cuda), _t(cents[i], cuda))
        torch.cuda.synchronize()
        assert torch.equal(b.cluster_labels_of(i).view(-1), one.cluster_labels), f"image {i}"
        assert torch.equal(b.centroids_of(i), one.centroids), f"image {i}"
        assert torch.equal(b.segment_labels_of(i).view(h, w), one.segment_labels), f"image {i}"


@pytest.mark.parametrize("w,h", [(64, 64), (131, 77), (4, 200)])
@pytest.mark.parametrize("policy", [0, 1])
def test_pipeline_without_erosion(cuda, w, h, policy):
    import torch
    from split_gb300 import pipeline
    rgb = synth.voronoi_rgb8(w, w, h, 12, sigma=14.0)
    pipe = pipeline.Pipeline(w, h, pipeline.Params(
        nclusters=6, dim=3, kmeans_iters=5, merge_P=30, merge_policy=policy, erode_radius=0,
        compute_normals=False), cuda)
    pipe.run(_t(rgb, cuda), _t(synth.pick_centroids(3, rgb, 6, 3), cuda))
    torch.cuda.synchronize()
    pipe.ws.check("pipeline")
    seg = oracle.ccl(pipe.cluster_labels.cpu().numpy().reshape(h, w), 8, 0)
    chroma = oracle.rgb_to_ic_f32(rgb)[1:] if policy else None
    assert np.array_equal(pipe.segment_labels.cpu().numpy(),
                          oracle.merge_small(seg, 30, policy, chroma))
