"""Smooth-boundary merge at the edges of its tiles and of their pair tables:
whole and ragged tiles, labels addressed at odd bytes of a line, more pairs
than a tile's table holds, one segment; equal to the oracle, twice through one
workspace."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,block,salt,offset", [
    ((32, 64), 16, 0.0, 0), ((33, 65), 12, 0.0, 1), ((31, 63), 9, 0.0, 3),
    ((70, 130), 33, 0.0, 2), ((96, 200), 7, 0.0, 0),
    ((64, 128), 32, 0.2, 0), ((65, 131), 40, 0.3, 2),   # single pixels: 1000 pairs a tile
    ((1, 300), 40, 0.0, 0), ((300, 1), 40, 0.0, 1), ((1, 1), 1, 0.0, 0), ((40, 70), 99, 0.0, 0)])
def test_merge_over_tiles(cuda, shape, block, salt, offset):
    import torch
    from split_gb300 import ccl
    h, w = shape
    rng = np.random.default_rng(100 * h + w)
    y, x = np.mgrid[0:h, 0:w]
    seg = (y // block * block * w + x // block * block).astype(np.int32)
    base = seg
    seg = np.where(rng.random((h, w)) < salt, y * w + x, seg).astype(np.int32)
    # classes whose mutual boundaries are smooth, other boundaries sharp
    pts = (rng.integers(0, 3, size=h * w)[base.ravel()] * 0.4
           + rng.random((3, h * w)) * 0.02).astype(np.float32)
    buf = torch.empty(h * w + 4, dtype=torch.int32, device=cuda)
    got = buf[offset:offset + h * w].view(h, w)
    got.copy_(torch.from_numpy(seg))
    dev = torch.from_numpy(pts).to(cuda)
    ws, ref = None, seg
    for threshold in (0.05, 2.0):
        ref = oracle.merge_smooth(ref, pts, threshold)
        ws = ccl.merge_smooth_boundaries(dev, 0, got, ws, threshold)
        ws.check("merge_smooth")
        assert np.array_equal(got.cpu().numpy(), ref)


def test_workspace_across_sizes(cuda):
    """One workspace for images of different sizes, back and forth."""
    import torch
    from split_gb300 import ccl
    ws = ccl.Workspace(ccl.merge_smooth_boundaries_workspace(300, 200), cuda)
    for w, h in ((300, 200), (70, 50), (290, 190), (300, 200), (128, 64), (300, 200)):
        rng = np.random.default_rng(w)
        y, x = np.mgrid[0:h, 0:w]
        seg = (y // 9 * 9 * w + x // 9 * 9).astype(np.int32)
        pts = (rng.integers(0, 3, size=h * w)[seg.ravel()] * 0.4
               + rng.random((3, h * w)) * 0.02).astype(np.float32)
        got = torch.from_numpy(seg).to(cuda)
        ccl.merge_smooth_boundaries(torch.from_numpy(pts).to(cuda), 0, got, ws, 0.05)
        ws.check("merge_smooth")
        assert np.array_equal(got.cpu().numpy(), oracle.merge_smooth(seg, pts, 0.05)), (w, h)
